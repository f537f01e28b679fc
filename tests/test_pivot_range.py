"""Pivots whose reciprocal is not a normal number.

The factorisations multiply by reciprocals of the pivots; a matrix scaled by
2^-130 has pivots in the subnormal range of FP32, whose reciprocals overflow,
one scaled by 2^-1030 the same in FP64.  Scaling matrix and right-hand side by
a power of two leaves the solution alone.

Mixed: FP32 keeps 2^-149 / 2^-130 = 2^-19 of the scaled entries, so the
preconditioner is good to about 2^-19 times the condition of a subdomain and
the iteration reaches 1e-5.  FP64: entries are rounded by 2^-45 of the
diagonal, times the condition number of the 8^3 problem (below 1e4, and a
factor of ten for the row sums): 1e-8.  One subdomain makes the FP64 solve a
direct one (r.r underflows, so one iteration is all there is).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPTS = dict(solver=2, method=1, fine_method=1, smoothers=1, strong1="0.08", radius1=2)


@pytest.mark.parametrize("scale", [0, -126, -128, -129, -130, 120])
def test_mixed_solve_of_a_scaled_matrix(scale):
    import doug_gb300 as D
    from doug_gb300 import problems as P
    n, r, c, v, b = P.diffusion3d_fv(12, seed=3)
    s = D.DougSolver(dict(OPTS, levels=2, overlap=1, solve_tolerance="1.0e-5", solve_maxiters=300, precision=1))
    s.set_matrix_coo(n, r, c, v * 2.0**scale)
    s.set_partition(P.block_partition(12, 2))
    s.setup()
    _, st = s.solve(b * 2.0**scale)
    assert st.true_rel_residual <= 1.001e-5


@pytest.mark.parametrize("panel_rows", [512, 16])
@pytest.mark.parametrize("scale", [0, -1022, -1030, 1000])
def test_fp64_solve_of_a_scaled_matrix(scale, panel_rows):
    import doug_gb300 as D
    from doug_gb300 import problems as P
    n, r, c, v, b = P.diffusion3d_fv(8, seed=3)
    a = np.zeros((n, n))
    np.add.at(a, (r - 1, c - 1), v)
    x = np.linalg.solve(a, b)
    s = D.DougSolver(dict(OPTS, levels=1, overlap=1, maxasize1=1000, solve_tolerance="1.0e-30", solve_maxiters=1,
                          precision=0, panel_rows=panel_rows, tensor_update=0))
    s.set_matrix_coo(n, r, c, np.ldexp(v, scale))
    s.set_partition(np.ones(n, np.int32))
    s.setup()
    got, _ = s.solve(np.ldexp(b, scale if scale <= 0 else 0), allow_not_converged=True)
    if scale > 0:
        got = np.ldexp(got, scale)
    assert np.linalg.norm(got - x) <= 1e-8 * np.linalg.norm(x)
