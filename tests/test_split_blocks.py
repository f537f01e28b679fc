"""The memory of the FP64 tensor-core updates' digit slices (split_blocks).

A super-panel step's fronts go in groups of at most split_blocks 64-row
blocks (128 KB each): a group's size changes launches and memory and nothing
else, so the solutions are bit-identical.  Without any (0, or where the device
has no memory left) the CUDA cores' kernel does the work, as with
tensor_update 0.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPTS = dict(solver=2, method=1, fine_method=1, levels=2, overlap=2, smoothers=1, strong1="0.08", radius1=2,
            solve_tolerance="1.0e-10", solve_maxiters=500, precision=0)


def _run(words, nrhs=1):
    import torch
    import doug_gb300 as D
    from doug_gb300 import problems as P
    n, r, c, v, b = P.diffusion3d_fv(30, seed=3)
    s = D.DougSolver(dict(OPTS, **words))
    s.set_matrix_coo(n, r, c, v)
    s.set_partition(P.block_partition(30, 2))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    s.setup()
    used = free - torch.cuda.mem_get_info()[0]
    x, st = s.solve(b) if nrhs == 1 else s.solve_multi(np.column_stack([b] * nrhs))
    return x, st, used


@pytest.mark.parametrize("nrhs", [1, 3])
def test_groups_change_launches_and_memory_only(nrhs):
    x, st, used = _run({}, nrhs)
    x40, st40, used40 = _run(dict(split_blocks=40), nrhs)
    x1, st1, _ = _run(dict(split_blocks=1), nrhs)
    assert np.array_equal(x, x1) and np.array_equal(x, x40)
    assert st.iterations == st1.iterations == st40.iterations
    assert st.gpu_launches < st40.gpu_launches < st1.gpu_launches
    assert used40 < used


def test_no_slices_is_the_cuda_core_update():
    x, st, _ = _run(dict(split_blocks=0))
    x0, st0, _ = _run(dict(tensor_update=0))
    assert np.array_equal(x, x0) and st.gpu_launches == st0.gpu_launches
