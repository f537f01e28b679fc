"""Which kernels factor a front, against the oracle.

A level of at least eight one-CTA fronts per SM goes to the one-CTA kernel,
a thinner one to the panel pipeline, whose panel step has one thread per row
with four CTAs per SM and more and four lanes per row below.  216 subdomains
of a 36^3 grid give levels of 6768 to 116 one-CTA fronts; panel_rows 16 sends
them all through the pipeline (both panel kernels); leaves of 65 and 97
pivots give panels of one pivot and of one row more than a CTA's 32.  Bars:
those of the other solve tests, FP64 1e-10 and mixed 1e-7 of the FP64 oracle
(tolerance 1e-12), the FP64 iteration count within one.
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
@pytest.mark.parametrize("n,parts,words", [(36, 6, {}), (36, 6, dict(panel_rows=16)),
                                           (13, 2, dict(nd_leaf=65, panel_rows=16)),
                                           (13, 2, dict(nd_leaf=97, panel_rows=16, super_panel=32))])
def test_factor_paths_match_the_oracle(n, parts, words, precision):
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
