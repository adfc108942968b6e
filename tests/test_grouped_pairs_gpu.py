"""The grouped tcgen05 product whose CTAs take two tiles of an expert: runs of one, two, three and more than 32 tiles (a warp looks
at 32 at a time), empty tiles between, lone tiles before another expert's and at the end."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("runs,N,K", [([(0, 1), (1, 3), (-1, 2), (2, 2), (0, 1), (1, 1), (2, 2)], 128, 64), ([(1, 33), (0, 64), (1, 1)], 256, 72),
                                      ([(0, 67)], 128, 520), ([(2, 2), (1, 2), (0, 2), (-1, 3), (1, 3)], 384, 1032)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_two_tiles_an_expert(runs, N, K, out_dtype):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(K)
    tiles = [e for e, n in runs for _ in range(n)]
    E, rows = 3, len(tiles) * ops.EXPERT_TILE
    assert len(tiles) >= 4 * E                            # many enough for the kernel under test
    x = torch.randn(rows, K, generator=gen, device=DEV).to(torch.bfloat16)
    w = torch.randn(E, N, K, generator=gen, device=DEV).to(torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = ops.grouped_linear(x, w, torch.tensor(tiles, dtype=torch.int32, device=DEV), out_dtype, err)
    assert int(err.item()) == 0
    for i, e in enumerate(tiles):
        if e < 0:
            continue
        a, b = x[i * 64:(i + 1) * 64].double(), w[e].double()
        bound = 2.0 ** -24 * K * (a.abs() @ b.abs().T) + (2.0 ** -8 * (a @ b.T).abs() if out_dtype == torch.bfloat16 else 0.0)
        assert bool(((out[i * 64:(i + 1) * 64].double() - a @ b.T).abs() <= bound).all()), i
