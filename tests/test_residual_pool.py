"""The scratch pool of dg_residual_csr keeps its memory over a synchronisation,
and no more than its bound; and a first call beside a capture, in the mode
that allows one.

Each in a process of its own, where the pool does not exist yet.
dg_residual_csr_noalloc runs first: it loads the same kernels and has no pool.
"""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

COMMON = """
import ctypes, sys
import torch
import doug_gb300 as D
L = D.load_library()
n = 100_000
ptr = torch.arange(n + 1, dtype=torch.int64, device="cuda")
col = torch.arange(n, dtype=torch.int32, device="cuda")
val, x, b = (torch.rand(n, dtype=torch.float64, device="cuda") for _ in range(3))
def call(f, r, s, stream):
    return f(n, *(t.data_ptr() for t in (ptr, col, val, x, b, r, s)), ctypes.c_void_p(stream.cuda_stream))
r0, r1, r2 = (torch.zeros_like(x) for _ in range(3))
s0, s1, s2 = (torch.zeros(1, dtype=torch.float64, device="cuda") for _ in range(3))
here = torch.cuda.current_stream()
assert call(L.dg_residual_csr_noalloc, r0, s0, here) == D.DG_OK
torch.cuda.synchronize()
"""

KEPT = COMMON + """
free = torch.cuda.mem_get_info()[0]
for _ in range(3):
    assert call(L.dg_residual_csr, r1, s1, here) == D.DG_OK
    torch.cuda.synchronize()
kept = free - torch.cuda.mem_get_info()[0]
assert torch.equal(r0, r1) and torch.equal(s0, s1)
assert 0 < kept <= 64 << 20, kept
"""

BESIDE = COMMON + """
side, other = torch.cuda.Stream(), torch.cuda.Stream()
g = torch.cuda.CUDAGraph()
# (relaxed: in the stricter modes an allocation on any stream breaks the capture)
with torch.cuda.graph(g, stream=side, capture_error_mode="relaxed"):
    assert call(L.dg_residual_csr, r1, s1, other) == D.DG_OK  # the pool is made here, on a stream that is not captured
    assert call(L.dg_residual_csr, r2, s2, side) == D.DG_OK
other.synchronize()
assert torch.equal(r0, r1) and torch.equal(s0, s1)
assert not torch.equal(r0, r2)
g.replay()
torch.cuda.synchronize()
assert torch.equal(r0, r2) and torch.equal(s0, s2)
"""


@pytest.mark.parametrize("script", [KEPT, BESIDE], ids=["kept", "beside_a_capture"])
def test_in_a_fresh_process(script):
    run = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
