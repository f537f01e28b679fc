"""The FP64 super-panel update on the tensor cores (tensor_update 1).

A dense matrix is one front, so one preconditioner step is its solve and the
first CG iterate's error is the factorisation's.  Sizes lie on both sides of
the tile (128 x 64), block (64) and super-panel (128, 64, 32) edges; one case
scales rows and columns by 2^-60 .. 2^60, one has rows that hold entries 2^-70
apart.  Bound: the matrices have condition at most 10 after scaling, so the
Cholesky solve's error is below 10 * n * eps relative, and the CG step's
scaling of it adds as much again: 20 n eps.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPTS = dict(solver=2, method=1, fine_method=1, levels=1, overlap=1, smoothers=1, strong1="0.08", radius1=2,
            solve_tolerance="1.0e-30", solve_maxiters=1, precision=0, nd_leaf=512, panel_rows=16,
            maxasize1=1000)


def _dense(n, kind):
    rng = np.random.default_rng(n)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (q * rng.uniform(1.0, 10.0, n)) @ q.T
    a = 0.5 * (a + a.T)
    if kind == "graded":  # off-diagonal entries over 70 binary orders, diagonally dominant
        a = rng.standard_normal((n, n)) * 2.0 ** -rng.integers(0, 70, (n, n))
        a = np.tril(a, -1)
        a = a + a.T
        a += np.diag(np.abs(a).sum(1) * 1.25 + 1.0)
        d = 1.0 / np.sqrt(np.diag(a))
        a = a * d * d[:, None]
    s = np.ones(n)
    if kind == "scaled":
        s = 2.0 ** rng.integers(-60, 61, n)
    x = rng.uniform(-1, 1, n)
    return a * s * s[:, None], x, s


@pytest.mark.parametrize("n,kind,words", [(33, "plain", {}), (129, "plain", {}), (161, "plain", dict(super_panel=32)),
                                          (192, "plain", dict(super_panel=64)), (193, "plain", {}), (256, "plain", {}),
                                          (257, "plain", {}), (330, "plain", {}), (500, "plain", {}),
                                          (290, "scaled", {}), (290, "graded", {})])
def test_dense_front_is_solved_to_fp64(n, kind, words):
    import doug_gb300 as D
    a, x, s = _dense(n, kind)
    b = (a.astype(np.longdouble) @ (x / s).astype(np.longdouble)).astype(np.float64)
    r, c = np.nonzero(np.ones((n, n)))
    sv = D.DougSolver(dict(OPTS, **words))
    sv.set_matrix_coo(n, r + 1, c + 1, a[r, c])
    sv.set_partition(np.ones(n, np.int32))
    sv.setup()
    got, st = sv.solve(b, allow_not_converged=True)
    assert st.nsubdomains == 1
    assert np.linalg.norm(got * s - x) <= 20 * n * 2.0**-53 * np.linalg.norm(x)
