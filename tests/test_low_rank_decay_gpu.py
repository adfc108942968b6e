"""Decays from a short product in one kernel: the bits of the product and the decay as kernels of their own, for ranks up to the one
it keeps (and one above, which takes the other two), ragged tokens and channels, rows of a wider matrix, with and without a bias."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T,N,rank,dtype,bias", [(1, 64, 16, torch.bfloat16, True), (17, 2048, 16, torch.bfloat16, True),
                                                 (33, 516, 16, torch.float32, True), (16, 515, 16, torch.bfloat16, False),
                                                 (40, 512, 13, torch.float32, True), (5, 7, 1, torch.bfloat16, True), (9, 128, 17, torch.bfloat16, True)])
def test_decays_of_a_short_product(T, N, rank, dtype, bias):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(T * N + rank)
    x = 6.0 * torch.randn(T, rank + 8, generator=gen, device=DEV)[:, 8:] if N != 515 else torch.randn(T, rank, generator=gen, device=DEV)
    w = torch.randn(N, rank, generator=gen, device=DEV).to(dtype)
    b = torch.randn(N, generator=gen, device=DEV) if bias else None
    x[0, 0], x[-1, -1] = float("inf"), -1e30
    z = torch.empty(T, N, device=DEV)
    want = ops.gated_decay(ops.gemm_f32_ex(x, w, z, T, N, rank, x.stride(0), N), b, 16.0)
    got = ops.low_rank_decay(x, w, b, 16.0)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    fin = torch.isfinite(x).all(1) & (x.abs() < 1e20).all(1)
    if bool(fin.any()):
        v = x[fin].double() @ w.double().T + (b.double() if bias else 0.0)
        bound = 2.0 ** -23 * (rank + 2) * (x[fin].double().abs() @ w.double().abs().T + (b.double().abs() if bias else 0.0)) / 16.0 + 2.0 ** -19
        ref = torch.exp(torch.nn.functional.logsigmoid(v) / 16.0)
        assert bool(((got[fin].double() - ref).abs() <= bound).all())
