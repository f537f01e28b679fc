"""Factors of a factorisation that timed out are not kept.

update_wait_polls 0 (a failure-test word) ends the FP64 tensor-core update of
a dense front early; reuse_factors would keep that factorisation.  Each solve
must report it, single, several right-hand sides and stacked systems alike,
and so must the setup of the robust coarse space, which factors its supports
(aggregates of 300 unknowns, a dense front each).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPTS = dict(solver=2, method=1, fine_method=1, levels=1, overlap=1, smoothers=1, strong1="0.08", radius1=2,
            solve_tolerance="1.0e-10", solve_maxiters=50, precision=0, nd_leaf=512, panel_rows=16, maxasize1=1000)


@pytest.mark.parametrize("form", ["single", "multi", "systems"])
def test_every_solve_reports_the_timeout(form):
    import doug_gb300 as D
    n = 290
    rng = np.random.default_rng(n)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (q * rng.uniform(1.0, 10.0, n)) @ q.T
    a = 0.5 * (a + a.T)
    r, c = np.nonzero(np.ones((n, n)))
    m = (n, (r + 1).astype(np.int32), (c + 1).astype(np.int32), a[r, c])
    s = D.DougSolver(dict(OPTS))
    s.set_option("update_wait_polls", 0)
    s.set_option("reuse_factors", 1)
    if form == "systems":
        s.set_systems([m, m])
    else:
        s.set_matrix_coo(*m)
        s.set_partition(np.ones(n, np.int32))
    s.setup()
    b = rng.uniform(-1, 1, 2 * n if form == "systems" else n)
    for _ in range(2):
        with pytest.raises(D.DougError) as e:
            s.solve_multi(np.column_stack([b, b[::-1]])) if form == "multi" else s.solve(b)
        assert e.value.status == D.DG_CUDA_ERROR and "factorisation" in str(e.value)


def test_robust_setup_reports_the_timeout():
    import doug_gb300 as D
    from doug_gb300 import problems as P
    n, r, c, v, _ = P.diffusion3d_fv(12, seed=4)
    s = D.DougSolver(dict(solver=2, method=1, fine_method=1, levels=2, overlap=1, smoothers=0, strong1="0.08", radius1=5,
                          coarse_method=2, maxasize1=300, nd_leaf=2000, solve_tolerance="1.0e-10",
                          solve_maxiters=500))
    s.set_option("update_wait_polls", 0)
    s.set_matrix_coo(n, r, c, v)
    with pytest.raises(D.DougError, match="timed out"):
        s.setup()
    s.set_option("update_wait_polls", -1)
    s.setup()
