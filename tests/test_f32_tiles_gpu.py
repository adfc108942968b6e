"""The tiled kernels of the 32-bit path give the bits of the simple ones: every output is a sum in one fixed order, whatever
the tile.  Products against the same product with its weights stored in bfloat16 (which takes the simple kernel), at the
edges of tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (5, 130, 20), (63, 64, 16), (65, 127, 44), (128, 4864, 32), (129, 4736, 36),
                                   (513, 2048, 68), (300, 20000, 8)])
def test_products_do_not_depend_on_the_tile(M, N, K):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(M + N)
    wide = torch.randn(M, K + 4, generator=gen, device=DEV)
    w = torch.randn(N, K, generator=gen, device=DEV).to(torch.bfloat16)
    for a, lda in ((wide[:, :K].contiguous(), K), (wide, K + 4)):
        for out_dtype in (torch.float32, torch.bfloat16):
            got, want = (torch.empty(M, N, dtype=out_dtype, device=DEV) for _ in range(2))
            ops.gemm_f32_ex(a, w.float(), got, M, N, K, lda, N)
            ops.gemm_f32_ex(a, w, want, M, N, K, lda, N)
            assert torch.equal(got, want)
    ref = wide[:, :K].double() @ w.double().T
    bound = (K + 1) * 2.0 ** -24 * (wide[:, :K].double().abs() @ w.double().abs().T)
    assert bool(((ops.gemm_f32(wide[:, :K].contiguous(), w.float()).double() - ref).abs() <= bound).all())


def test_gathered_rows_batches_and_weights_per_tile():
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(3)
    M, N, K, E = 200, 136, 52, 3
    a = torch.randn(90, K, generator=gen, device=DEV)
    w = torch.randn(E, N, K, generator=gen, device=DEV).to(torch.bfloat16)
    rows = torch.randint(-1, 90, (M,), generator=gen, device=DEV, dtype=torch.int32)
    tile_w = torch.tensor([2, -1, 0, 1], dtype=torch.int32, device=DEV)
    outs = [torch.zeros(M, N, device=DEV) for _ in range(2)]
    for out, ww in zip(outs, (w.float(), w)):
        ops.gemm_f32_ex(a, ww, out, M, N, K, K, N, w_bs=N * K, a_rows=rows, tile_w=tile_w)
    assert torch.equal(*outs) and bool((outs[0][64:128] == 0).all())
    x = torch.randn(70, E, K, generator=gen, device=DEV)                      # a batch per head, rows of a wider tensor
    outs = [torch.zeros(70, E, N + 8, device=DEV) for _ in range(2)]
    for out, ww in zip(outs, (w.float(), w)):
        ops.gemm_f32_ex(x, ww, out, 70, N, K, E * K, E * (N + 8), batch=E, a_bs=K, w_bs=N * K, c_bs=N + 8)
    assert torch.equal(*outs) and bool((outs[0][:, :, N:] == 0).all())
