"""dg_residual_csr over its lane widths and block edges.

A block of rows takes 1, 4, 16 or 32 lanes per row by its average row length,
256 or 1,024 rows per block by the system's size: each width, a last block of
one row, empty rows and the larger block size, against a plain FP64 product.
Tolerance: a row of k entries is k fused multiply-adds and at most 5 shuffle
additions, so |r - r_ref| <= (k + 8) 2^-52 (|A||x| + |b|) row by row, the
reference's own sum included twice over; the norm is a sum of n squares.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(1, 1), (255, 3), (257, 12), (256, 13), (1025, 40), (513, 60), (300, 200), (260, 500),
                                 (1_228_801, 5)])
def test_residual_matches_plain_product(n, k):
    torch = pytest.importorskip("torch")
    import doug_gb300 as D
    rng = np.random.default_rng(n + k)
    length = np.full(n, min(k, n))
    length[rng.random(n) < 0.1] = 0  # empty rows
    ptr = np.concatenate([[0], np.cumsum(length)]).astype(np.int64)
    col = rng.integers(0, n, ptr[-1]).astype(np.int32)
    val = rng.uniform(-1, 1, ptr[-1])
    x, b = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    t = [torch.tensor(a, device="cuda") for a in (ptr, col, val, x, b)]
    r, nrm = D.residual_csr(*t)
    row = np.repeat(np.arange(n), length)
    ref = b - np.bincount(row, val * x[col], minlength=n)
    bound = (k + 8) * 2.0 ** -52 * (np.bincount(row, np.abs(val * x[col]), minlength=n) + np.abs(b))
    got = r.cpu().numpy()
    assert np.all(np.abs(got - ref) <= 2 * bound)
    assert abs(nrm.item() - got @ got) <= (n + 8) * 2.0 ** -52 * (got @ got)


def test_residual_under_capture_and_beside_it():
    torch = pytest.importorskip("torch")
    import doug_gb300 as D
    n = 1000
    ptr = torch.arange(n + 1, dtype=torch.int64, device="cuda")
    col = torch.arange(n, dtype=torch.int32, device="cuda")
    val, x, b = (torch.rand(n, dtype=torch.float64, device="cuda") for _ in range(3))
    ref, _ = D.residual_csr(ptr, col, val, x, b)
    L = D.load_library()
    r, s = torch.zeros_like(x), torch.zeros(1, dtype=torch.float64, device="cuda")
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        stream = torch.cuda.current_stream().cuda_stream
        assert L.dg_residual_csr(n, *(t.data_ptr() for t in (ptr, col, val, x, b, r, s)), ctypes.c_void_p(stream)) == D.DG_OK
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(r, ref)
