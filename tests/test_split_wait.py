"""The FP64 tensor-core update when its epilogue's wait runs out.

update_wait_polls 0 (a failure-test word) makes every epilogue warp give up
at once, while the copies and products of the tile go on and are waited for.
The status reaches the host, whether a CTA has one tile (a dense front of 290)
or a second one follows (1600); the handle recovers with the usual limit.
Bound of the solve: that of the dense-front tests, 20 n eps.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPTS = dict(solver=2, method=1, fine_method=1, levels=1, overlap=1, smoothers=1, strong1="0.08", radius1=2,
            solve_tolerance="1.0e-30", solve_maxiters=1, precision=0, nd_leaf=2000, panel_rows=16, maxasize1=2000)


def dense(n):
    rng = np.random.default_rng(n)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (q * rng.uniform(1.0, 10.0, n)) @ q.T
    a = 0.5 * (a + a.T)
    x = rng.uniform(-1, 1, n)
    b = (a.astype(np.longdouble) @ x.astype(np.longdouble)).astype(np.float64)
    return a, x, b


@pytest.mark.parametrize("n", [290, 1600])
def test_epilogue_timeout_is_reported(n):
    import doug_gb300 as D
    a, x, b = dense(n)
    r, c = np.nonzero(np.ones((n, n)))
    s = D.DougSolver(dict(OPTS))
    s.set_option("update_wait_polls", 0)
    s.set_matrix_coo(n, r + 1, c + 1, a[r, c])
    s.set_partition(np.ones(n, np.int32))
    s.setup()
    with pytest.raises(D.DougError) as e:
        s.solve(b, allow_not_converged=True)
    assert e.value.status == D.DG_CUDA_ERROR and "timed out" in str(e.value)
    s.set_option("update_wait_polls", -1)
    s.setup()
    got, _ = s.solve(b, allow_not_converged=True)
    assert np.linalg.norm(got - x) <= 20 * n * 2.0**-53 * np.linalg.norm(x)
