"""Joined levels of the assembly tree against the oracle.

Short levels are joined (up to four into one): a front then holds a separator
and its descendants and has four, eight or sixteen children instead of two,
which the solves take in pairs, four at once, or one by one.  Leaves of 2 and
3 unknowns give deep trees (joins of four levels), thin_level_fronts 0 none,
100000 joins of long levels too (warp kernels never); one subdomain joins
less than many.  Bars: those of the other solve tests, FP64 1e-10 and mixed
1e-7 of the FP64 oracle (tolerance 1e-12), the FP64 iteration count within one.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "oracle"))

pytestmark = pytest.mark.gpu

OPTS = dict(solver=2, method=1, fine_method=1, levels=2, overlap=2, smoothers=1, strong1="0.08", radius1=2,
            solve_tolerance="1.0e-12", solve_maxiters=500)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dim,n,parts,words", [(2, 33, 1, {}), (2, 60, 3, {}), (2, 47, 2, dict(nd_leaf=2)),
                                               (3, 12, 1, dict(nd_leaf=3)), (3, 20, 2, {}),
                                               (3, 20, 2, dict(thin_level_fronts=0)),
                                               (3, 20, 3, dict(thin_level_fronts=100000)),
                                               (3, 20, 3, dict(thin_level_fronts=100000, lean_task_kb=1)),
                                               (3, 14, 2, dict(nd_leaf=4, solve_schedule=1))])
def test_joined_levels_match_the_oracle(dim, n, parts, words, precision):
    import doug_gb300 as D
    import oracle as O
    from doug_gb300 import problems as P
    if dim == 2:
        nn, r, c, v, b, _ = P.poisson2d_p1(n + 2, seed=n)
    else:
        nn, r, c, v, b = P.diffusion3d_fv(n, seed=n + parts)
    side = round(nn ** (1.0 / dim))
    assert side**dim == nn
    part = P.block_partition(side, parts, dim)
    ro = O.run_coo(nn, r, c, v, rhs=b, ctl="".join(f"{k} {x}\n" for k, x in OPTS.items()), part=part)
    s = D.DougSolver(dict(OPTS, precision=precision, **words))
    s.set_matrix_coo(nn, r, c, v)
    s.set_partition(part)
    s.setup()
    x, st = s.solve(b)
    assert np.linalg.norm(x - ro["x"]) <= (1e-10 if precision == 0 else 1e-7) * np.linalg.norm(ro["x"])
    if precision == 0:
        assert abs(st.iterations - ro["iterations"]) <= 1
    X, _ = s.solve_multi(np.column_stack([b[::-1], b, b]))
    assert np.linalg.norm(X[:, 1] - x) <= (1e-10 if precision == 0 else 1e-7) * np.linalg.norm(x)
