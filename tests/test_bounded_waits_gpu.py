"""What kernels do when a bounded wait runs out: a block that leaves early waits for its copies first, and the delta rule's walk
says so and leaves the states as they were."""
import ctypes
import hashlib
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


@pytest.mark.parametrize("d,e,lens", [(128, 32, [65, 1, 200]), (64, 16, [64])])
def test_a_walk_that_gives_up_leaves_the_states(d, e, lens, monkeypatch):
    """The barrier of the first chunk waits for more bytes than come; the kernels that do not wait run to their end."""
    from ai_engine_b200.csrc.build import CSRC, cuda_library
    from ai_engine_b200.kernels import ops
    from test_linear_recurrence_chunked_gpu import Ctx
    with open(os.path.join(CSRC, "delta_rule_parallel.cu"), "rb") as f:      # (a source that another includes is not in its key)
        key = hashlib.sha256(f.read()).hexdigest()[:8]
    lib = ctypes.CDLL(cuda_library(os.path.join(HERE, "delta_walk_gives_up.cu"), [f"-DSOURCE_KEY=0x{key}"]))
    monkeypatch.setattr(ops, "library", lambda name, f=ops.library: lib if name == "delta_rule_parallel.cu" else f(name))
    monkeypatch.setattr(ops, "DELTA_PARALLEL_CHUNKS", 1)
    gen = torch.Generator(device=DEV).manual_seed(d)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    H, T = 2, sum(lens)
    rows, state = rnd(T, 2 * H * d + H * e), rnd(len(lens) + 1, H, d, e)
    ctx = Ctx(lens, list(range(len(lens))))
    ctx.live, before = None, state.clone()
    ops.delta_rule(rows[:, :H * d], rows[:, H * d:2 * H * d], rows[:, 2 * H * d:], rnd(T, H), rnd(T, H), rnd(H), rnd(H), d ** -0.5, 1e-6,
                   state, ctx, H, H, d, e, chunked=True)
    assert int(ctx.err.item()) == 4                                   # a bounded wait ran out, and nothing else
    long = [i for i, n in enumerate(lens) if n >= 64]
    assert torch.equal(state[long], before[long]) and torch.equal(state[-1], before[-1])
