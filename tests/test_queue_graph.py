"""Single solves of the dependency-driven schedule before and after several
right-hand sides: the captured iteration holds the queue's done flags, which a
larger number of right-hand sides allocates anew."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_single_multi_single(precision):
    import doug_gb300 as D
    from doug_gb300 import problems as P
    n, r, c, v, b = P.diffusion3d_fv(14, seed=9)
    s = D.DougSolver(dict(solver=2, method=1, fine_method=1, levels=2, overlap=2, smoothers=1, strong1="0.08", radius1=2,
                          solve_tolerance="1.0e-10", solve_maxiters=300, precision=precision))
    s.set_option("solve_schedule", 1)
    s.set_matrix_coo(n, r, c, v)
    s.set_partition(P.block_partition(14, 2))
    s.setup()
    x, st = s.solve(b)
    for k in (3, 7, 2):
        s.solve_multi(np.column_stack([b] * k))
        again, st2 = s.solve(b)
        assert np.array_equal(x, again) and st2.iterations == st.iterations
