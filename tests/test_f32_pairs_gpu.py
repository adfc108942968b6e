"""The three forms of the 32-bit product (narrow tiles, the same with lines asked for early, wide tiles) give the bits of the simple
kernel: every output is one sum over k in order.  The simple kernel takes the same weights stored in bfloat16; sizes lie at the
edges of tiles of rows (16, 32 and 64 of them in the last one), columns and k, and on either side of the rule between the forms."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M,N,K", [
    (1, 64, 4), (33, 66, 12), (64, 9472, 16),                            # narrow, one block an SM or fewer
    (40, 19000, 20), (257, 4800, 140), (96, 18944, 36),                  # narrow, more of them
    (65, 18941, 44), (80, 16384, 16), (81, 16386, 52), (96, 37888, 20), (129, 16383, 148), (192, 18944, 32)])   # wide
def test_every_form_gives_the_simple_kernel_s_bits(M, N, K):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(M * 7 + K)
    a = torch.randn(M, K, generator=gen, device=DEV)
    w = torch.randn(N, K, generator=gen, device=DEV).to(torch.bfloat16)
    for out_dtype, ldc in ((torch.float32, N), (torch.float32, N + 4), (torch.bfloat16, N + 1)):
        got, want = (torch.zeros(M, ldc, dtype=out_dtype, device=DEV) for _ in range(2))
        ops.gemm_f32_ex(a, w.float(), got, M, N, K, K, ldc)
        ops.gemm_f32_ex(a, w, want, M, N, K, K, ldc)
        assert torch.equal(got, want) and bool((got[:, N:] == 0).all())


def test_rows_that_are_left_out_and_values_that_are_not_finite():
    """An entry of -1 is a row of zeros; infinities and NaN reach the outputs of their own row and column alone."""
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(5)
    for M, N, K in ((70, 130, 36), (129, 16384, 20)):
        a = torch.randn(M, K, generator=gen, device=DEV)
        a[3, 7], a[M - 1, K - 1] = float("inf"), float("nan")
        w = torch.randn(N, K, generator=gen, device=DEV).to(torch.bfloat16)
        w[N - 1, 0] = -float("inf")
        rows = torch.randint(0, M, (M,), generator=gen, device=DEV, dtype=torch.int32)
        rows[1], rows[M - 1] = -1, 3
        got, want = (torch.zeros(M, N, device=DEV) for _ in range(2))
        ops.gemm_f32_ex(a, w.float(), got, M, N, K, K, N, a_rows=rows)
        ops.gemm_f32_ex(a, w, want, M, N, K, K, N, a_rows=rows)
        assert torch.equal(got.nan_to_num(nan=1e30, posinf=2e30, neginf=3e30), want.nan_to_num(nan=1e30, posinf=2e30, neginf=3e30))
        assert bool((got[1, :N - 1] == 0).all()) and not bool(torch.isfinite(got[M - 1]).any())
