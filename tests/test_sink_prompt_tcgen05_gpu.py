"""The tcgen05 prompt kernel with kept first keys, a factor, a distance bias, a sink and a gate per head, against the formula
in 64 bits on the same bfloat16 rows: windows that start inside and at the edges of pages and key tiles, kept keys that end
inside a page, fill tiles of their own and reach into the window, pages that the window has passed and that are gone."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def reference(q, rows, reqs, temp, slope, sink, gate, scale, window, keep):
    """q [T, H, d] and rows per request [n, G, 2 d] in float64: outputs and sums of weights times |value|."""
    T, H, d = q.shape
    out, mag, at = torch.empty_like(q), torch.empty_like(q), 0
    for (c, n), r in zip(reqs, rows):
        i, j = torch.arange(c, c + n, device=DEV)[:, None], torch.arange(c + n, device=DEV)[None, :]
        ok = j <= i
        if window:
            ok &= (i - j < window) | (j < keep)
        for h in range(H):
            k, v = r[:, h * r.shape[1] // H, :d], r[:, h * r.shape[1] // H, d:]
            s = (q[at:at + n, h] @ k.T) * (scale * (temp[h] if temp is not None else 1.0))
            if slope is not None:
                s = s - slope[h] * (i - j)
            s = s.masked_fill(~ok, -float("inf"))
            m = s.amax(1, keepdim=True)
            if sink is not None:
                m = torch.maximum(m, sink[h])
            p = torch.exp(s - m)
            p = p / (p.sum(1, keepdim=True) + (torch.exp(sink[h] - m) if sink is not None else 0.0))
            g = gate[at:at + n, h, None] if gate is not None else 1.0
            out[at:at + n, h], mag[at:at + n, h] = g * (p @ v), g * (p @ v.abs())
        at += n
    return out, mag


@pytest.mark.parametrize("H,G,d,P,reqs,window,keep,extras", [
    (4, 2, 128, 16, [(0, 64), (900, 130), (0, 1), (3, 5)], 300, 4, "tslg"),
    (2, 1, 128, 8, [(1000, 200)], 128, 130, "sl"), (2, 2, 64, 16, [(2000, 300), (40, 129)], 257, 400, "tslg"),
    (3, 1, 64, 128, [(700, 140)], 1, 1, "lg"), (2, 1, 128, 32, [(500, 260)], 100, 600, "ts"),
    (2, 2, 128, 16, [(0, 300), (129, 128)], 0, 7, "tslg"), (1, 1, 64, 64, [(1300, 128)], 640, 0, "l")])
def test_prompts_with_kept_keys_bias_sink_and_gate(H, G, d, P, reqs, window, keep, extras, monkeypatch):
    from ai_engine_b200.cache import PagedCache
    from ai_engine_b200.engine.step import StepContext, StepEntry
    from ai_engine_b200.kernels import ops
    from ai_engine_b200.parts import ATTENTION_WORK, CacheNeed, KVRequest
    gen = torch.Generator(device=DEV).manual_seed(window * 7 + d + H)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    cache = PagedCache([CacheNeed(0, "m", KVRequest(G, 2 * d, window, planes=1, keep_first=keep if window else 0))], P,
                       sum(-(-(c + n) // P) for c, n in reqs) + 2, len(reqs), 4096, torch.bfloat16, DEV)
    entries, rows, pool = [], [], cache.groups[0].pool                    # unwritten places hold NaN
    for c, n in reqs:
        s = cache.admit()
        cache.ensure(s, c + n)
        entries.append(StepEntry(s, c, [0] * n, []))
        rows.append(rnd(c + n, G, 2 * d).to(torch.bfloat16))
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    ctx = StepContext(entries, cache, torch.device(DEV), err, planners=(ATTENTION_WORK,))
    lc = cache.layer_cache(0, ctx)["m"]
    bt = lc.block_table.clone()
    host = bt.cpu()
    for r, (c, n) in enumerate(reqs):
        for pg in range(-(-(c + n) // P)):
            first, last = pg * P, min((pg + 1) * P, c + n)
            if window and last <= c - window + 1 and first >= keep:
                bt[r, pg] = -1                                            # passed by the window of every query: gone
                continue
            pool[0, 0, int(host[r, pg]), :, :last - first] = rows[r][first:last].transpose(0, 1)
    q = rnd(sum(n for _, n in reqs), H, d).to(torch.bfloat16)
    temp = rnd(H) if "t" in extras else None                             # factors below zero among them
    slope = 2.0 ** -torch.arange(1, H + 1, device=DEV).float() if "l" in extras else None
    sink = 2.0 * rnd(H) if "s" in extras else None
    gate = torch.sigmoid(rnd(q.shape[0], H)) if "g" in extras else None
    took, real = [], ops.paged_attention_prefill_rows
    monkeypatch.setattr(ops, "paged_attention_prefill_rows", lambda *a, **k: took.append(real(*a, **k)) or took[-1])
    args = (q, lc.k_pages, gate, temp, slope, sink, ctx, ctx.plan(ATTENTION_WORK), bt, d, d ** -0.5, window, keep)
    got = ops.sink_attention(*args)
    assert took == [True] and int(err.item()) == 0
    f64 = lambda t: t.double() if t is not None else None
    ref, mag = reference(q.double(), [r.double() for r in rows], reqs, f64(temp), f64(slope), f64(sink), f64(gate), d ** -0.5,
                         window, keep)
    # one rounding to bfloat16; weights of 16 bits; scores of up to 2^10 in float32 (2^-14 in the exponent, a few times)
    assert bool(((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -11 * mag + 1e-6).all())
    monkeypatch.setattr(ops, "paged_attention_prefill_rows", lambda *a, **k: False)
    other = ops.sink_attention(*args)
    assert bool(((other.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -11 * mag + 1e-6).all())
