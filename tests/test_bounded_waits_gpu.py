"""What kernels do when a bounded wait runs out: a block that leaves early waits for its copies first."""
import ctypes
import os

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("stages,asked", [(1, 1), (1, 2), (2, 1), (2, 2), (2, 3), (3, 7), (4, 4), (4, 9), (6, 17), (8, 8), (8, 31), (4, 0)])
@pytest.mark.parametrize("late", [0, 30000, -1])
def test_a_block_that_leaves_early_waits_for_its_copies(stages, asked, late):
    """Each stage's last copy is in flight for `late` cycles (-1: it never comes, and the wait for it ends all the same)."""
    from ai_engine_b200.csrc.build import cuda_library
    lib = ctypes.CDLL(cuda_library(os.path.join(HERE, "bounded_waits.cu")))
    src = torch.arange(1, 4 * 64 + 1, dtype=torch.int32, device=DEV)
    out = torch.full((8,), -7, dtype=torch.int32, device=DEV)
    assert lib.late_copies(ctypes.c_void_p(src.data_ptr()), ctypes.c_void_p(out.data_ptr()), stages, asked, ctypes.c_longlong(late),
                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    last = [max((i for i in range(asked) if i % stages == s), default=None) for s in range(stages)]
    assert out.tolist() == [0 if i is None or late < 0 else 4 * i + 1 for i in last] + [-7] * (8 - stages)
