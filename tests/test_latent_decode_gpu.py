"""Lone tokens over the compressed cache: the kernel that cuts the visible rows of all requests into equal stretches, against
the formula in 64 bits on the same bfloat16 rows.  Requests of one key, of a chunk more or less, longer than a stretch and by
the dozen in one; windows; heads that fill part of a tile or more than one; rows of odd sizes; short portions beside them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("H,rank,rot,P,reqs,window,sink,exact", [
    (16, 512, 64, 16, [(c, 1) for c in (0, 1, 31, 32, 33, 700, 2000, 63, 64, 5, 129)], 0, True, False),
    (3, 64, 16, 8, [(7 * i % 40, 1) for i in range(70)], 0, False, True),           # many requests in a stretch
    (18, 192, 32, 16, [(3000, 1)], 0, True, True),                                  # one request over many stretches
    (5, 128, 0, 32, [(900, 1), (10, 1), (300, 1)], 100, False, False), (1, 320, 48, 16, [(500, 1), (0, 1)], 1, True, False),
    (8, 64, 80, 16, [(40, 1), (3, 7), (200, 1), (0, 2), (77, 1)], 64, False, True), (16, 448, 576, 16, [(65, 1), (1000, 1)], 0, False, False),
    (4, 192, 576, 16, [(65, 1), (30, 3), (1000, 1), (0, 9)], 0, True, False)])             # rows too long for the portions' kernel
def test_lone_tokens(H, rank, rot, P, reqs, window, sink, exact, monkeypatch):
    from ai_engine_b200.cache import PagedCache
    from ai_engine_b200.engine.step import StepContext, StepEntry
    from ai_engine_b200.kernels import ops
    from ai_engine_b200.parts import LATENT_WORK, CacheNeed, KVRequest
    gen = torch.Generator(device=DEV).manual_seed(rank + len(reqs))
    dk = rank + rot
    cache = PagedCache([CacheNeed(0, "m", KVRequest(1, dk, 0, planes=1))], P, sum(-(-(c + n) // P) for c, n in reqs) + 2,
                       len(reqs), 4096, torch.bfloat16, DEV)
    entries, rows, pool = [], [], cache.groups[0].pool                    # unwritten places hold NaN
    for c, n in reqs:
        s = cache.admit()
        cache.ensure(s, c + n)
        entries.append(StepEntry(s, c, [0] * n, []))
        rows.append(torch.randn(c + n, dk, generator=gen, device=DEV).to(torch.bfloat16))
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    ctx = StepContext(entries, cache, torch.device(DEV), err, planners=(LATENT_WORK,))
    lc = cache.layer_cache(0, ctx)["m"]
    host = lc.block_table.cpu()
    for r, (c, n) in enumerate(reqs):
        for j in range(c + n):
            pool[0, 0, int(host[r, j // P]), 0, j % P] = rows[r][j]
    T = sum(n for _, n in reqs)
    q = torch.randn(T, H, dk, generator=gen, device=DEV).to(torch.bfloat16).float()
    sinks = torch.randn(H, generator=gen, device=DEV) if sink else None
    scale = 1.5 * dk ** -0.5
    lib, ran = ops.library("latent_attention_tc.cu"), []
    entry = lambda *a: ran.append(1) or lib.aie_latent_decode(*a)
    fake = type("Lib", (), dict(aie_latent_decode=staticmethod(entry), aie_latent_attention_tc=lib.aie_latent_attention_tc))
    monkeypatch.setattr(ops, "library", lambda name, f=ops.library: fake if name == "latent_attention_tc.cu" else f(name))
    got = ops.latent_attention(q, lc.k_pages, ctx, lc.block_table, rank, scale, window, torch.bfloat16, ctx.plan(LATENT_WORK),
                               sink=sinks, exact_weights=exact)
    assert int(err.item()) == 0 and ran == [1]                            # lone tokens have their kernel in every step
    at = 0
    for (c, n), rr in zip(reqs, rows):
        k = rr.double()
        for i in range(n):
            p, lo = c + i, max(c + i - window + 1, 0) if window else 0
            s = q[at].double() @ k[lo:p + 1].T * scale
            m = s.amax(1, keepdim=True) if sinks is None else torch.maximum(s.amax(1, keepdim=True), sinks.double()[:, None])
            w = torch.exp(s - m)
            w = w / (w.sum(1, keepdim=True) + (torch.exp(sinks.double()[:, None] - m) if sinks is not None else 0.0))
            ref, mag = w @ k[lo:p + 1, :rank], w @ k[lo:p + 1, :rank].abs()
            # the result rounded once; weights of 8 bits, or of 16
            bound = 2.0 ** -8 * ref.abs() + (2.0 ** -14 if exact else 2.0 ** -8) * mag
            assert bool(((got[at].double() - ref).abs() <= bound).all()), (c, i)
            at += 1
