"""dg_residual_csr on long rows among short ones.

A row of more than 64 times its block's lanes per row is summed by a whole
warp: one long row at either end of a block, many of them, all lanes-per-row
widths, rows at the limit and one entry above it.  Tolerance as for ordinary
rows: k entries are k fused multiply-adds and at most 5 shuffle additions,
the reference's own sum included twice over.
"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(length, seed=0):
    rng = np.random.default_rng(seed)
    n = len(length)
    ptr = np.concatenate([[0], np.cumsum(length)]).astype(np.int64)
    col = rng.integers(0, n, ptr[-1]).astype(np.int32)
    return ptr, col, rng.uniform(-1, 1, ptr[-1]), rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)


@pytest.mark.parametrize("n,short,long,where", [(256, 7, 1200, [0]), (256, 7, 1200, [255]), (700, 2, 65, range(0, 700, 29)),
                                                (700, 2, 64, range(0, 700, 29)), (1000, 0, 3000, [511, 512, 999]),
                                                (600, 20, 257, range(5, 600, 50)), (600, 20, 4000, [300, 301, 302]),
                                                (520, 100, 1025, [3, 260]), (520, 100, 1024, [3, 260]),
                                                (520, 100, 9000, [519])])
def test_long_rows(n, short, long, where):
    torch = pytest.importorskip("torch")
    import doug_gb300 as D
    length = np.full(n, short)
    length[list(where)] = long
    a = _matrix(length, n + long)
    ptr, col, val, x, b = a
    r, nrm = D.residual_csr(*[torch.tensor(t, device="cuda") for t in a])
    row = np.repeat(np.arange(n), length)
    ref = b - np.bincount(row, val * x[col], minlength=n)
    bound = (length + 8) * 2.0**-52 * (np.bincount(row, np.abs(val * x[col]), minlength=n) + np.abs(b))
    got = r.cpu().numpy()
    assert np.all(np.abs(got - ref) <= 2 * bound)
    assert abs(nrm.item() - got @ got) <= (n + 8) * 2.0**-52 * (got @ got)


def test_one_long_row_does_not_hold_up_the_rest():
    """200,000 rows of 7, one of 1,200: a warp's 10 rounds of loads beside
    10 MB; a single lane's 300 rounds took four times as long as the rest."""
    torch = pytest.importorskip("torch")
    import doug_gb300 as D
    best = []
    for long in (7, 1200):
        length = np.full(200_000, 7)
        length[100_000] = long
        t = [torch.tensor(q, device="cuda") for q in _matrix(length)]
        times = []
        for _ in range(5):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for _ in range(200):
                D.residual_csr(*t)
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t0)
        best.append(min(times))
    assert best[1] < 2 * best[0]
