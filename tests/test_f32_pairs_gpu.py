"""The three forms of the 32-bit product (narrow tiles, the same with lines asked for early, wide tiles) give the bits of the simple
kernel: every output is one sum over k in order.  The simple kernel takes the same weights stored in bfloat16; sizes lie at the
edges of tiles of rows (16, 32 and 64 of them in the last one), columns and k, and on either side of the rule between the forms;
gathered rows, batches and weights per tile of rows in each form."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


NARROW, AHEAD, WIDE = 0, 1, 2


def form_of(M, N, batch=1):
    from ai_engine_b200.kernels import ops
    return ops.library("gemm_f32.cu").aie_gemm_f32_form(M, N, batch, ops.sm_count())


def test_the_sizes_below_reach_every_form():
    for form, sizes in ((AHEAD, [(1, 64), (33, 66), (64, 9472), (1, 2048), (33, 130), (64, 4736), (7, 64)]),
                        (NARROW, [(40, 19000), (257, 4800), (80, 16384), (81, 16386), (96, 37888)]),
                        (WIDE, [(96, 18944), (65, 18941), (129, 16383), (192, 18944), (80, 18944), (144, 16384), (81, 18944), (145, 14208)])):
        assert all(form_of(M, N) == form for M, N in sizes)
    assert form_of(70, 130, 3) == AHEAD and form_of(70, 4736, 3) == WIDE and form_of(144, 2048, 4) == WIDE and form_of(70, 2048, 8) == NARROW


@pytest.mark.parametrize("M,N,K", [
    (1, 64, 4), (33, 66, 12), (64, 9472, 16),                            # one block an SM or fewer
    (1, 2048, 132), (33, 130, 1028), (64, 4736, 144), (7, 64, 2052),     # ... and long enough that lines are asked for early
    (40, 19000, 20), (257, 4800, 140), (80, 16384, 16), (81, 16386, 52), (96, 37888, 20),       # narrow, more blocks
    (65, 18941, 44), (96, 18944, 36), (129, 16383, 148), (192, 18944, 32),                      # wide: 1, 32, 1 and 64 rows in the last tile,
    (80, 18944, 52), (144, 16384, 20), (81, 18944, 148), (145, 14208, 16)])                     # 16 and 17
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


@pytest.mark.parametrize("M,N,K,batch", [(70, 130, 164, 3), (70, 4736, 36, 3), (144, 2048, 52, 4), (70, 2048, 20, 8)])
def test_batches(M, N, K, batch):
    """Products side by side, rows and results of wider tensors."""
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(M + N)
    x = torch.randn(M, batch, K, generator=gen, device=DEV)
    w = torch.randn(batch, N, K, generator=gen, device=DEV).to(torch.bfloat16)
    for pad in (8, 1):                                                   # stores of 16 bytes and of one element
        got, want = (torch.zeros(M, batch, N + pad, device=DEV) for _ in range(2))
        for out, ww in ((got, w.float()), (want, w)):
            ops.gemm_f32_ex(x, ww, out, M, N, K, batch * K, batch * (N + pad), batch=batch, a_bs=K, w_bs=N * K, c_bs=N + pad)
        assert torch.equal(got, want) and bool((got[:, :, N:] == 0).all())


@pytest.mark.parametrize("M,N,K", [(200, 136, 164), (192, 18944, 36), (209, 8192, 20), (150, 9472, 20)])
def test_weights_per_tile_of_rows_and_gathered_rows(M, N, K):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(M)
    a = torch.randn(90, K, generator=gen, device=DEV)
    w = torch.randn(3, N, K, generator=gen, device=DEV).to(torch.bfloat16)
    rows = torch.randint(-1, 90, (M,), generator=gen, device=DEV, dtype=torch.int32)
    tile_w = torch.tensor([2, -1, 0, 1], dtype=torch.int32, device=DEV)[:(M + 63) // 64]
    got, want = (torch.zeros(M, N, device=DEV) for _ in range(2))
    for out, ww in ((got, w.float()), (want, w)):
        ops.gemm_f32_ex(a, ww, out, M, N, K, K, N, w_bs=N * K, a_rows=rows, tile_w=tile_w)
    assert torch.equal(got, want) and bool((got[64:128] == 0).all())
    ref = a.double()[rows.long()[128:]] @ w[0].double().T                 # (the third tile's weight)
    n = min(64, M - 128)
    bound = (K + 1) * 2.0 ** -24 * (a.double().abs()[rows.long()[128:]] @ w[0].double().abs().T)
    ok = ((got[128:].double() - ref).abs() <= bound)[:n] | (rows[128:128 + n, None] < 0)
    assert bool(ok.all())
