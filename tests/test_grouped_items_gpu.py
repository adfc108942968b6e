"""The grouped tcgen05 product whose blocks walk items of up to four tiles of an expert: runs of one to nine and more than 32 tiles,
empty tiles between, more items than SMs, a remainder of K, one block an item and two; with and without the gated unit, which gives the bits of the unit on
the float32 product."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("runs,N,K", [
    ([(0, 1), (1, 3), (-1, 2), (2, 2), (0, 4), (1, 5), (2, 9)], 128, 64), ([(1, 33), (0, 65), (1, 1)], 256, 72), ([(-1, 3)], 128, 64),
    ([(2, 1)], 384, 520), ([(0, 7), (-1, 1), (2, 6), (1, 40)], 1152, 1032),
    ([(0, 7), (-1, 1), (2, 6), (1, 40)], 1280, 1032), ([(-1, 3)], 256, 1024), ([(2, 1)], 256, 1024)])
def test_items_of_up_to_four_tiles(runs, N, K):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(K + N)
    tiles = [e for e, n in runs for _ in range(n)]
    rows = len(tiles) * ops.EXPERT_TILE
    x = torch.randn(rows, K, generator=gen, device=DEV).to(torch.bfloat16)
    w = torch.randn(3, N, K, generator=gen, device=DEV).to(torch.bfloat16)
    tile_w = torch.tensor(tiles, dtype=torch.int32, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    outs = {}
    for dtype in (torch.float32, torch.bfloat16):
        out = outs[dtype] = torch.full((rows, N), 7.0, dtype=dtype, device=DEV)
        ops._grouped_items(x, w, tile_w, out, err, None, None)
        for i, e in enumerate(tiles):
            got = out[i * 64:(i + 1) * 64].double()
            if e < 0:
                assert bool((got == 7.0).all())                      # skipped tiles are left as they are
                continue
            a, b = x[i * 64:(i + 1) * 64].double(), w[e].double()
            bound = 2.0 ** -24 * K * (a.abs() @ b.abs().T) + (2.0 ** -8 * (a @ b.T).abs() if dtype == torch.bfloat16 else 0.0)
            assert bool(((got - a @ b.T).abs() <= bound).all()), (dtype, i)
    live = (tile_w >= 0).repeat_interleave(64)
    for limit, alpha, shift in ((float("inf"), 1.0, 0.0), (7.0, 1.702, 1.0)):
        got = ops.grouped_glu(x, w, tile_w, limit, alpha, shift, torch.bfloat16, err, None)
        want = ops.clamped_glu(outs[torch.float32], N // 2, limit, alpha, shift, torch.bfloat16)
        assert torch.equal(got[live], want[live])
    assert int(err.item()) == 0


def test_more_tiles_than_the_list_holds_take_the_other_kernels():
    from ai_engine_b200.kernels import ops
    tiles = ops.GROUPED_MAX_TILES + 1
    gen = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn(tiles * 64, 64, generator=gen, device=DEV).to(torch.bfloat16)
    w = torch.randn(1, 128, 64, generator=gen, device=DEV).to(torch.bfloat16)
    tile_w = torch.zeros(tiles, dtype=torch.int32, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    act = ops.grouped_glu(x, w, tile_w, float("inf"), 1.0, 0.0, torch.bfloat16, err, torch.arange(tiles * 64, dtype=torch.int32, device=DEV))
    gu = x.double() @ w[0].double().T
    want = torch.nn.functional.silu(gu[:, :64]) * gu[:, 64:]
    assert bool(((act.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -16 * gu.abs().amax()).all()) and int(err.item()) == 0
