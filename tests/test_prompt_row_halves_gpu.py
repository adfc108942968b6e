"""The tcgen05 prompt kernel with two threads a query row: a row's maximum that moves from one key tile to the next, in the first or
the second 64 keys of a tile, by more than the reference follows and by less, and rows whose first tiles hold nothing they read
(a window, kept keys alone), with one query, whole tiles and a remainder.  Against the formula in 64 bits."""
import pytest
import torch

from test_sink_prompt_tcgen05_gpu import reference

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("reqs,window,keep", [([(700, 129), (0, 2)], 0, 0), ([(383, 257)], 200, 0), ([(1000, 128), (130, 33)], 129, 3)])
@pytest.mark.parametrize("step", [3.0, 40.0])
def test_maxima_that_move_in_either_half(d, reqs, window, keep, step):
    from ai_engine_b200.cache import PagedCache
    from ai_engine_b200.engine.step import StepContext, StepEntry
    from ai_engine_b200.kernels import ops
    from ai_engine_b200.parts import ATTENTION_WORK, CacheNeed, KVRequest
    gen = torch.Generator(device=DEV).manual_seed(int(step) + d + window)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    H, G, P = 2, 1, 16
    cache = PagedCache([CacheNeed(0, "m", KVRequest(G, 2 * d, 0, planes=1))], P, sum(-(-(c + n) // P) for c, n in reqs), len(reqs),
                       4096, torch.bfloat16, DEV)
    entries, rows, pool = [], [], cache.groups[0].pool
    for c, n in reqs:
        s = cache.admit()
        cache.ensure(s, c + n)
        entries.append(StepEntry(s, c, [0] * n, []))
        r = 0.25 * rnd(c + n, G, 2 * d)
        # element 0 of the keys climbs by `step` every 64 keys and falls back after seven, so scores do (queries have 1 there)
        at = torch.arange(c + n, device=DEV) // 64
        r[:, 0, 0] = step * (at % 7)
        rows.append(r.to(torch.bfloat16))
    ctx = StepContext(entries, cache, torch.device(DEV), torch.zeros(1, dtype=torch.int32, device=DEV), planners=(ATTENTION_WORK,))
    lc = cache.layer_cache(0, ctx)["m"]
    bt = lc.block_table.cpu()
    for r, (c, n) in enumerate(reqs):
        for pg in range(-(-(c + n) // P)):
            first, last = pg * P, min((pg + 1) * P, c + n)
            pool[0, 0, int(bt[r, pg]), :, :last - first] = rows[r][first:last].transpose(0, 1)
    q = rnd(sum(n for _, n in reqs), H, d)
    q[:, :, 0] = 1.0
    q = q.to(torch.bfloat16)
    out = torch.empty_like(q)
    assert ops.paged_attention_prefill_rows(q, lc.k_pages, ctx.plan(ATTENTION_WORK), ctx, lc.block_table, 1.0, window, 0.0, False,
                                            None, out, keep_first=keep)
    assert int(ctx.err.item()) == 0
    lone = torch.cat([torch.full((n,), n == 1, device=DEV) for _, n in reqs])
    ref, mag = reference(q.double(), [r.double() for r in rows], reqs, None, None, None, None, 1.0, window, keep)
    # one rounding to bfloat16; weights of 16 bits; scores below 2^8 in float32 (2^-16 in the exponent, a few times)
    ok = (out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -12 * mag + 1e-6
    assert bool(ok[~lone].all())
