"""The level solves' kernel variants against the oracle.

A level of fronts is solved by warp kernels (many small fronts) or by CTA
tasks in one of four variants per direction, chosen by the number and length
of its tasks.  64 subdomains of an irregular 3-D grid give levels on both
sides of every line: warp kernels and one wave of short tasks by default;
every front as CTA tasks (thin_level_fronts) gives the 128-thread variants,
with lean_task_kb 1 the 256-thread one; leaves of 3 unknowns give tiny fronts
and fronts of more than two children; one subdomain gives the longest fronts.
The last four reach the ends of the one-CTA factorisation: leaves of 2, 33 and
90 pivots, and every front of more than 20 rows through the panel pipeline.
Bars: those of the other solve tests, FP64 1e-10 and mixed 1e-7 of the FP64
oracle (tolerance 1e-12), the FP64 iteration count within one.
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
@pytest.mark.parametrize("n,parts,words", [(26, 4, {}), (26, 4, dict(thin_level_fronts=100000)),
                                           (26, 4, dict(thin_level_fronts=100000, lean_task_kb=1)),
                                           (26, 4, dict(thin_level_fronts=0)), (17, 2, dict(nd_leaf=3)),
                                           (21, 1, dict(fwd_task_kb=1)), (11, 2, dict(nd_leaf=2)),
                                           (19, 2, dict(nd_leaf=33)), (19, 2, dict(nd_leaf=90)),
                                           (21, 1, dict(panel_rows=20))])
def test_variants_match_the_oracle(n, parts, words, precision):
    import doug_gb300 as D
    import oracle as O
    from doug_gb300 import problems as P
    nn, r, c, v, b = P.diffusion3d_fv(n, seed=n + parts)
    part = P.block_partition(n, parts)
    ro = O.run_coo(nn, r, c, v, rhs=b, ctl="".join(f"{k} {x}\n" for k, x in OPTS.items()), part=part)
    s = D.DougSolver(dict(OPTS, precision=precision, **words))
    s.set_matrix_coo(nn, r, c, v)
    s.set_partition(part)
    s.setup()
    x, st = s.solve(b)
    assert np.linalg.norm(x - ro["x"]) <= (1e-10 if precision == 0 else 1e-7) * np.linalg.norm(ro["x"])
    if precision == 0:
        assert abs(st.iterations - ro["iterations"]) <= 1
    B = np.column_stack([b, b[::-1], np.arange(nn) % 7 - 3.0])
    X, _ = s.solve_multi(B)
    assert np.linalg.norm(X[:, 0] - x) <= (1e-10 if precision == 0 else 1e-7) * np.linalg.norm(x)
