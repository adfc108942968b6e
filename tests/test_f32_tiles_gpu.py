"""The tiled kernels of the 32-bit path give the bits of the simple ones: every output is a sum in one fixed order, whatever
the tile.  Products against the same product with its weights stored in bfloat16 (which takes the simple kernel),
attention against the plain kernel, at the edges of tiles, chunks, pages and windows."""
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


@pytest.mark.parametrize("H,K,d,P,reqs,window", [
    (4, 2, 64, 16, [(0, 64), (0, 65), (70, 1)], 0), (2, 1, 128, 8, [(100, 130), (5, 8)], 0), (3, 3, 20, 4, [(127, 9), (0, 200)], 0),
    (2, 2, 96, 16, [(300, 70), (0, 1), (128, 2)], 100), (1, 1, 4, 2, [(0, 257)], 1), (8, 1, 32, 32, [(1, 127), (129, 129)], 64)])
def test_attention_of_portions_has_the_plain_kernel_s_bits(H, K, d, P, reqs, window):
    from ai_engine_b200.cache import PagedCache
    from ai_engine_b200.engine.step import StepContext, StepEntry
    from ai_engine_b200.kernels import ops
    from ai_engine_b200.parts import ATTENTION_WORK, CacheNeed, KVRequest
    gen = torch.Generator(device=DEV).manual_seed(H * 10 + d)
    cache = PagedCache([CacheNeed(0, "m", KVRequest(K, d))], P, sum(-(-(c + n) // P) for c, n in reqs) + 2, len(reqs), 4096,
                       torch.float32, DEV)
    entries, pool = [], cache.groups[0].pool                               # unwritten places hold NaN
    for c, n in reqs:
        s = cache.admit()
        cache.ensure(s, c + n)
        entries.append(StepEntry(s, c, [0] * n, []))
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    ctx = StepContext(entries, cache, torch.device(DEV), err, planners=(ATTENTION_WORK,))
    lc = cache.layer_cache(0, ctx)["m"]
    bt = lc.block_table.cpu().numpy()
    for r, (c, n) in enumerate(reqs):
        for j in range(c + n):
            pool[0, :, int(bt[r, j // P]), :, j % P] = torch.randn(2, K, d, generator=gen, device=DEV)
    q = torch.randn(sum(n for _, n in reqs), H, d, generator=gen, device=DEV)
    got = ops.paged_attention(q, lc.k_pages, lc.v_pages, ctx, ctx.plan(ATTENTION_WORK), lc.block_table, 0.3, window)
    want = ops.paged_attention_plain(q, lc.k_pages, lc.v_pages, ctx.positions, ctx.token_req, lc.block_table, 0.3, window, err)
    assert torch.equal(got, want) and not bool(got.isnan().any()) and int(err.item()) == 0
    bad = lc.block_table.clone()                                          # a page outside the pool is flagged and skipped
    bad[0, 0] = pool.shape[2] + 7
    got = ops.paged_attention(q, lc.k_pages, lc.v_pages, ctx, ctx.plan(ATTENTION_WORK), bad, 0.3, 0)
    assert int(err.item()) == 2
    want = ops.paged_attention_plain(q, lc.k_pages, lc.v_pages, ctx.positions, ctx.token_req, bad, 0.3, 0, err)
    assert torch.equal(got, want)


def step(H, K, d, P, reqs, seed=1):
    """A step over filled pages: (ctx, cache, queries)."""
    from ai_engine_b200.cache import PagedCache
    from ai_engine_b200.engine.step import StepContext, StepEntry
    from ai_engine_b200.parts import ATTENTION_WORK, CacheNeed, KVRequest
    gen = torch.Generator(device=DEV).manual_seed(seed)
    cache = PagedCache([CacheNeed(0, "m", KVRequest(K, d))], P, sum(-(-(c + n) // P) for c, n in reqs), len(reqs), 4096, torch.float32, DEV)
    entries = []
    for c, n in reqs:
        s = cache.admit()
        cache.ensure(s, c + n)
        entries.append(StepEntry(s, c, [0] * n, []))
    cache.groups[0].pool.normal_(generator=gen)
    ctx = StepContext(entries, cache, torch.device(DEV), torch.zeros(1, dtype=torch.int32, device=DEV), planners=(ATTENTION_WORK,))
    return ctx, cache.layer_cache(0, ctx)["m"], torch.randn(sum(n for _, n in reqs), H, d, generator=gen, device=DEV)


def both(ctx, lc, q, window):
    from ai_engine_b200.kernels import ops
    from ai_engine_b200.parts import ATTENTION_WORK
    return (ops.paged_attention(q, lc.k_pages, lc.v_pages, ctx, ctx.plan(ATTENTION_WORK), lc.block_table, 0.3, window),
            ops.paged_attention_plain(q, lc.k_pages, lc.v_pages, ctx.positions, ctx.token_req, lc.block_table, 0.3, window, ctx.err))


@pytest.mark.parametrize("window", [0, 40, 129])
@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan")])
@pytest.mark.parametrize("plane", [0, 1])
def test_keys_and_values_that_are_not_finite_reach_the_queries_that_see_them(plane, value, window):
    ctx, lc, q = step(4, 2, 64, 16, [(0, 150), (200, 70)])
    planes = (lc.k_pages, lc.v_pages)[plane]
    for r, at in ((0, 3), (0, 63), (0, 131), (1, 20), (1, 150), (1, 233)):
        planes[int(lc.block_table[r, at // 16]), :, at % 16, ::5] = value
    got, want = both(ctx, lc, q, window)
    assert bool(torch.isfinite(want).any()) and not bool(torch.isfinite(want).all())
    assert torch.equal(got.nan_to_num(nan=1e30, posinf=2e30, neginf=3e30), want.nan_to_num(nan=1e30, posinf=2e30, neginf=3e30))


def test_operands_off_the_16_byte_grid_take_the_plain_kernel():
    ctx, lc, q = step(2, 1, 20, 4, [(3, 70), (0, 9)])
    off = lambda t: torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view(t.shape)
    got, want = both(ctx, lc, off(q), 0)
    assert torch.equal(got, want)
    planes = type("Planes", (), dict(k_pages=lc.k_pages, v_pages=off(lc.v_pages), block_table=lc.block_table))
    got, want = both(ctx, planes, q, 33)
    assert torch.equal(got, want) and int(ctx.err.item()) == 0
