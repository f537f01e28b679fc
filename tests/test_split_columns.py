"""The FP64 tensor-core update at every number of columns.

Two dense leaves of a and b unknowns meet in a dense separator of s: each
leaf's front is one super-panel of a (b) columns with s update rows, so that
split_always gives updates of any number of columns: one chunk of 64 or two,
remainders of the 16 columns of a product, both leaves in one launch.  The
separator's front (s pivots) has full super-panels and a last one without rows
below.  s = 2000 gives each leaf 408 tiles, several to a CTA.  narrow
super-panels give 32 and 64 columns in a front of 161 and 193.

The launches tell that the path is taken: two a step instead of one.  One
subdomain and one iteration make the solve a direct one; matrices of condition
below 10: 20 n eps, as for a dense front.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPTS = dict(solver=2, method=1, fine_method=1, levels=1, overlap=1, smoothers=1, strong1="0.08", radius1=2,
            solve_tolerance="1.0e-30", solve_maxiters=1, precision=0, panel_rows=16, maxasize1=100000,
            thin_level_fronts=0)


def two_leaves(a, b, s, seed=0):
    """(n, rows0, cols0, vals): leaves [0, a) and [a, a + b), separator behind; the first node of a leaf of more than
    one has no neighbour in the separator, so that the dissection's levels are leaf, separator, leaf."""
    rng = np.random.default_rng(seed + 1000 * a + b)
    n = a + b + s
    m = rng.uniform(-1, 1, (n, n))
    m = np.tril(m, -1)
    m[a:a + b, :a] = 0
    for p, k in ((0, a), (a, b)):
        if k > 1:
            m[a + b:, p] = 0
    m = m + m.T
    m += np.diag(np.abs(m).sum(1) * 1.5)
    d = 1 / np.sqrt(np.diag(m))
    m = m * d[:, None] * d
    r, c = np.nonzero(m)
    return n, r, c, m[r, c]


def run(n, r, c, v, **words):
    import doug_gb300 as D
    x = np.random.default_rng(n).uniform(-1, 1, n)
    b = np.add.reduceat(v.astype(np.longdouble) * x[c], np.searchsorted(r, np.arange(n))).astype(np.float64)
    s = D.DougSolver(dict(OPTS, **words))
    s.set_matrix_coo(n, r + 1, c + 1, v)
    s.set_partition(np.ones(n, np.int32))
    s.setup()
    got, st = s.solve(b, allow_not_converged=True)
    return np.linalg.norm(got - x) / np.linalg.norm(x), st.gpu_launches


@pytest.mark.parametrize("a,b,s", [(1, 1, 70), (15, 17, 100), (16, 32, 129), (31, 48, 90), (63, 64, 70), (65, 64, 128),
                                   (80, 81, 130), (100, 128, 257), (127, 128, 66), (17, 128, 400), (128, 128, 2000),
                                   (40, 100, 1000)])
def test_leaves_of_any_number_of_columns(a, b, s):
    m = two_leaves(a, b, s)
    words = dict(nd_leaf=max(a, b, 2))
    err, launches = run(*m, split_always=1, **words)
    cuda, plain = run(*m, tensor_update=0, **words)
    n = m[0]
    assert cuda <= 20 * n * 2.0**-53
    assert err <= 20 * n * 2.0**-53
    assert launches > plain


@pytest.mark.parametrize("n,words", [(161, dict(super_panel=32)), (193, dict(super_panel=64)), (97, dict(super_panel=32)),
                                     (193, {})])
def test_narrow_super_panels(n, words):
    m = two_leaves(1, 1, n - 2)
    err, launches = run(*m, split_always=1, nd_leaf=2, **words)
    _, plain = run(*m, tensor_update=0, nd_leaf=2, **words)
    assert err <= 20 * n * 2.0**-53
    assert launches > plain


def test_rows_with_an_infinity_are_not_positive_definite():
    """Pivots of 1e-290 under entries of 1e160 give rows of L beyond the largest number: the update's result is NaN,
    the separator's pivots are not positive, and the solve says so."""
    import doug_gb300 as D
    n, r, c, v = two_leaves(40, 40, 130)
    v = np.where((r >= 80) != (c >= 80), v * 1e160, v)
    v = np.where((r < 80) & (c < 80), v * 1e-290, v)
    s = D.DougSolver(dict(OPTS, split_always=1, nd_leaf=40))
    s.set_matrix_coo(n, r + 1, c + 1, v)
    s.set_partition(np.ones(n, np.int32))
    s.setup()
    with pytest.raises(D.DougError) as e:
        s.solve(np.ones(n), allow_not_converged=True)
    assert e.value.status == D.DG_SINGULAR
