"""A subdomain whose nodes lie far apart in the numbering, against the oracle.

The subdomain analysis looks nodes up by an array over the subdomain's range
of nodes, and in a sorted list where that range is more than 32 times its
size: the first part holds the first and the last five of 3,844 unknowns, the
others are contiguous.  Bars: those of the other solve tests.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "oracle"))

pytestmark = pytest.mark.gpu

OPTS = dict(solver=2, method=1, fine_method=1, levels=2, overlap=1, smoothers=1, strong1="0.08", radius1=2,
            solve_tolerance="1.0e-12", solve_maxiters=500)


@pytest.mark.parametrize("precision", [0, 1])
def test_far_nodes_in_one_subdomain(precision):
    import doug_gb300 as D
    import oracle as O
    from doug_gb300 import problems as P
    n, r, c, v, b, _ = P.poisson2d_p1(64, seed=5)
    part = (2 + np.arange(n) // 500).astype(np.int32)
    part[:5] = part[-5:] = 1
    ro = O.run_coo(n, r, c, v, rhs=b, ctl="".join(f"{k} {x}\n" for k, x in OPTS.items()), part=part)
    s = D.DougSolver(dict(OPTS, precision=precision))
    s.set_matrix_coo(n, r, c, v)
    s.set_partition(part)
    s.setup()
    x, st = s.solve(b)
    assert np.linalg.norm(x - ro["x"]) <= (1e-10 if precision == 0 else 1e-7) * np.linalg.norm(ro["x"])
    if precision == 0:
        assert abs(st.iterations - ro["iterations"]) <= 1
