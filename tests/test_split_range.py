"""FP64 tensor-core updates near the ends of the exponent range.

A dense matrix of condition below 10 as one front: the solve with its factor
is good to 20 n eps (see the dense-front test), whatever power of two scales
the matrix.  At 2^-1015 the products of the update lie around the smallest
normal number, where the sums keep 2^-59 of the diagonal; at 2^1015 the
matrix is solved for an unscaled right-hand side.  r.r underflows in the first
case: one iteration is all there is.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPTS = dict(solver=2, method=1, fine_method=1, levels=1, overlap=1, smoothers=1, strong1="0.08", radius1=2,
            solve_tolerance="1.0e-30", solve_maxiters=1, precision=0, nd_leaf=512, panel_rows=16, maxasize1=1000)


@pytest.mark.parametrize("scale", [0, -1015, 1015])
def test_scaled_dense_front(scale):
    import doug_gb300 as D
    n = 290
    rng = np.random.default_rng(n)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (q * rng.uniform(1.0, 10.0, n)) @ q.T
    a = 0.5 * (a + a.T)
    x = rng.uniform(-1, 1, n)
    b = (a.astype(np.longdouble) @ x.astype(np.longdouble)).astype(np.float64)
    r, c = np.nonzero(np.ones((n, n)))
    s = D.DougSolver(dict(OPTS))
    s.set_matrix_coo(n, r + 1, c + 1, np.ldexp(a[r, c], scale))
    s.set_partition(np.ones(n, np.int32))
    s.setup()
    got, _ = s.solve(np.ldexp(b, min(scale, 0)), allow_not_converged=True)
    got = np.ldexp(got, max(scale, 0))
    assert np.linalg.norm(got - x) <= 20 * n * 2.0**-53 * np.linalg.norm(x)
