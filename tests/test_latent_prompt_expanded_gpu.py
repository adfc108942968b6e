"""Latent attention of prompt portions over expanded rows: against the plain implementation in 64 bits and beside the path
that reads rows as they are (whose error it must not exceed), with windows at the edges of key tiles and pages, portions at
the edges of its query tiles and of the shortest it takes, and requests beside them that are too short for it."""
import pytest
import torch

import plain_vatazen as pv
from test_vatazen_parts_gpu import DT, Rig, f64, latent_part, lm, rnd, yarn
from zupitar_helpers import load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,rank,page,window,scaling", [(2, 64, 16, None, None), (3, 128, 8, 200, yarn(4.0, 100, 8.0, 0.5)),
                                                            (1, 512, 32, 129, None), (2, 256, 16, 64, yarn(16.0, 64))])
def test_portions_over_expanded_rows(heads, rank, page, window, scaling, monkeypatch):
    from ai_engine_b200.kernels import ops
    hidden, lens = 128, (420, 64, 200, 90)
    cuts = [[129, 64, 1, 128, 63, 35], [64], [1, 130, 2, 67], [63, 27]]
    # queries of deviation 0.3 sqrt(128) on keys of 0.3 sqrt(rank): scores of about 1.5.  A score's relative error (a rounded
    # query on a rounded key, or its latent form: 2^-9 each) is then an error of 1.5 x 2^-8.5 in the exponent
    m = lm(heads, 128, 64, 128, rank, 1.5 / (0.3 * 128 ** 0.5 * 0.3 * rank ** 0.5 * 128 ** 0.5), window, 20000.0, scaling)
    gen = torch.Generator().manual_seed(rank + (window or 0))
    part, t = latent_part(m, hidden, 1e-5, "bfloat16", gen)
    load(part, {k: v.to(torch.bfloat16) for k, v in t.items()}, torch.bfloat16)
    assert part.w_expand is not None
    seqs = [rnd(gen, n, hidden) for n in lens]
    refs = [pv.latent_attention(s.double(), f64(t), "", m, 1e-5) for s in seqs]
    calls, real = [], ops.latent_prompt
    monkeypatch.setattr(ops, "latent_prompt", lambda *a, **k: calls.append(a[6]) or real(*a, **k))
    run = lambda: Rig(part, DT["bfloat16"], page=page, pages=-(-sum(lens) // page) + 8).run([s.to(torch.bfloat16) for s in seqs], cuts)
    got = run()
    assert len(calls) == 3                                   # steps with a portion of 64 or more
    monkeypatch.setattr(ops, "LATENT_EXPAND_BYTES", 0)      # no room: every row is read as it is
    folded = run()
    assert len(calls) == 3
    errors = [[float(((o - r).norm() / r.norm())) for o, r in zip(os, refs)] for os in (got, folded)]
    # 1.5 x 2^-8.5 from the scores, and latents, values, outputs and their projection of 2^-9 / sqrt(3) each
    assert max(errors[0]) <= 6 * 2.0 ** -9, errors
    assert sum(errors[0]) <= 1.05 * sum(errors[1]), errors     # 5 %: what the errors of two draws of roundings differ by


def test_a_page_outside_the_pool_is_flagged():
    from ai_engine_b200.kernels import ops
    gen = torch.Generator().manual_seed(1)
    m = lm(1, 128, 64, 128, 64, 0.1, None)
    part, t = latent_part(m, 128, 1e-5, "bfloat16", gen)
    load(part, {k: v.to(torch.bfloat16) for k, v in t.items()}, torch.bfloat16)
    rig = Rig(part, DT["bfloat16"], page=16, pages=16)
    slot = rig.admit()
    ctx, lc = rig.step([(slot, 70)])
    lc.block_table = lc.block_table.clone()
    lc.block_table[0, 2] = 99
    part.forward(rnd(gen, 70, 128).to(torch.bfloat16).cuda(), ctx, lc)
    assert int(rig.err.item()) == 2


def test_tokens_beside_a_prompt_are_the_only_ones_that_are_folded(monkeypatch):
    """Four decoded tokens and a short portion beside two prompts: the products that fold and unfold see their rows alone, and
    every request has the bits that it has in a step of its own kind."""
    from ai_engine_b200.kernels import ops
    gen = torch.Generator().manual_seed(4)
    m = lm(2, 128, 64, 128, 64, 0.1, None)
    part, t = latent_part(m, 128, 1e-5, "bfloat16", gen)
    load(part, {k: v.to(torch.bfloat16) for k, v in t.items()}, torch.bfloat16)
    rows_seen, real = [], ops.head_linear
    monkeypatch.setattr(ops, "head_linear", lambda x, w, out: rows_seen.append(x.shape[0]) or real(x, w, out))
    before, brings = (40, 0, 7, 300, 20, 0, 99), (1, 100, 1, 1, 7, 70, 1)
    seqs = [rnd(gen, c + n, 128).to(torch.bfloat16).cuda() for c, n in zip(before, brings)]

    def run(groups):
        rig = Rig(part, DT["bfloat16"], page=16, pages=64, max_seqs=8)
        slots, out = [rig.admit() for _ in seqs], {}

        def step(who, rows):
            portions = [(slots[i], len(x)) for i, x in zip(who, rows)]
            ctx, lc = rig.step(portions)
            got = part.forward(torch.cat(rows), ctx, lc)
            rig.done(portions)
            return (got.sum(0) if got.dim() == 3 else got).split([len(x) for x in rows])

        for i, c in enumerate(before):
            if c:
                step([i], [seqs[i][:c]])
        rows_seen.clear()
        for who in groups:
            out.update(zip(who, step(who, [seqs[i][before[i]:] for i in who])))
        return [out[i] for i in range(len(seqs))], list(rows_seen)

    together, seen = run([list(range(7))])
    assert seen == [11, 11]                                       # 1 + 1 + 1 + 7 + 1
    apart, _ = run([[0, 2, 3, 6], [4], [1, 5]])
    for a, b in zip(together, apart):
        # the joins of parts and the output's product follow the step's shape: bfloat16 roundings of equal sums
        assert float((a.float() - b.float()).abs().max()) <= 2.0 ** -6 * float(b.float().abs().max())


@pytest.mark.parametrize("window", [None, 100])
def test_expanded_rows_have_a_bound_and_no_bit_depends_on_it(window, monkeypatch):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator().manual_seed(6)
    m = dict(lm(5, 128, 64, 128, 64, 0.1, window))
    part, t = latent_part(m, 128, 1e-5, "bfloat16", gen)
    load(part, {k: v.to(torch.bfloat16) for k, v in t.items()}, torch.bfloat16)
    seqs, cuts = [rnd(gen, n, 128).to(torch.bfloat16) for n in (200, 70, 300, 90)], [[200], [70], [130, 170], [5, 85]]
    products, real = [], ops.linear
    monkeypatch.setattr(ops, "linear", lambda x, w, *a: products.append((w.shape[0] % 320 == 0 and x.shape[0] % 128 == 0
                                                                       and x.shape[1] == 128, x.shape[0] * w.shape[0] * 2)) or real(x, w, *a))
    run = lambda: Rig(part, DT["bfloat16"], page=16, pages=64).run(seqs, cuts)
    want, most = run(), max(size for mine, size in products if mine)
    for bound in (most // 2, 128 * 640 * 3, 1):
        monkeypatch.setattr(ops, "LATENT_EXPAND_BYTES", bound)
        products.clear()
        got = run()
        sizes = [size for mine, size in products if mine]
        assert len(sizes) > 2 and max(sizes) <= max(bound, 3 * 128 * 640)            # three tiles: the longest portion, one head
        assert all(torch.equal(a, b) for a, b in zip(want, got))
    monkeypatch.setattr(ops, "LATENT_EXPAND_BYTES", 1 << 28)
    full = [3]                                                    # no room for three products: fewer heads at a time

    def tight(x, w, *a):
        if w.shape[0] > 320 and w.shape[0] % 320 == 0 and x.shape[0] % 128 == 0 and full[0]:
            full[0] -= 1
            raise torch.OutOfMemoryError("no room")
        return real(x, w, *a)

    monkeypatch.setattr(ops, "linear", tight)
    assert all(torch.equal(a, b) for a, b in zip(want, run())) and full[0] < 3


def test_a_query_latent_a_gate_a_head_and_a_rotation_of_halves(monkeypatch):
    """The other design's layer: queries through a latent of their own, a gate a head, pairs half a rotation apart, no sink and
    softmax weights of 8 bits where rows are read as they are."""
    import plain_fokisun as pf
    from ai_engine_b200.kernels import ops
    from test_fokisun_parts_gpu import latent_part as gated_part
    gen = torch.Generator().manual_seed(8)
    m = dict(heads=3, dim=128, rot_dim=64, vdim=128, kv_rank=128, q_rank=72, scale=0.004, rot=dict(base=20000.0, dims=64))
    part, t = gated_part(m, 96, 1e-5, "bfloat16", gen)
    load(part, {k: v.to(torch.bfloat16) for k, v in t.items()}, torch.bfloat16)
    assert part.w_expand is not None and part.halves and part.head_gate and part.q_rank and not part.exact_weights
    seqs, cuts, calls, real = [rnd(gen, n, 96) for n in (300, 150)], [[200, 1, 99], [3, 64, 83]], [], ops.latent_prompt
    refs = [pf.latent_attention(s.double(), f64(t), "", m, 1e-5) for s in seqs]
    monkeypatch.setattr(ops, "latent_prompt", lambda *a, **k: calls.append(1) or real(*a, **k))
    run = lambda: Rig(part, DT["bfloat16"], page=16, pages=64).run([s.to(torch.bfloat16) for s in seqs], cuts)
    got = run()
    assert len(calls) == 3
    monkeypatch.setattr(ops, "LATENT_EXPAND_BYTES", 0)
    folded = run()
    errors = [[float((o - r).norm() / r.norm()) for o, r in zip(os, refs)] for os in (got, folded)]
    # scores of about 1: 2^-8.5 of them in the exponent; queries' latent, latents, values, gate, outputs and their projection 2^-9 each
    assert len(calls) == 3 and max(errors[0]) <= 6 * 2.0 ** -9 and sum(errors[0]) <= 1.05 * sum(errors[1]), errors


def test_a_layer_that_reads_another_s_cache(monkeypatch):
    from ai_engine_b200.kernels import ops
    from test_pifutar_parts_gpu import latent_part as sharing_part, latent_tensors
    gen = torch.Generator().manual_seed(3)
    m = dict(heads=2, dim=128, rot_dim=64, vdim=128, kv_rank=64, scale=0.05, rot=dict(base=10000.0, dims=64))
    ts = latent_tensors(torch.bfloat16, 64, m, gen)
    owner = load(sharing_part(torch.bfloat16, 64, m, False), ts, torch.bfloat16)
    reader = load(sharing_part(torch.bfloat16, 64, m, True), {k: v for k, v in ts.items() if not k.startswith("dkv")}, torch.bfloat16)
    rig, h = Rig(owner, torch.bfloat16, page=16, pages=32), torch.randn(230, 64, generator=gen).to(torch.bfloat16).cuda()
    slot, at = rig.admit(), 0
    for n in (130, 100):
        ctx, lc = rig.step([(slot, n)])
        want = owner.forward(h[at:at + n], ctx, lc)
        pages = lc.k_pages.clone()
        got = reader.forward(h[at:at + n], ctx, lc)                # the same weights: the same rows, which it must not write
        a, b = (o.sum(0) if o.dim() == 3 else o for o in (got, want))
        assert float((a.float() - b.float()).abs().max()) <= 2.0 ** -6 * float(b.float().abs().max())      # queries by another product
        assert torch.equal(pages.nan_to_num(7.0), lc.k_pages.nan_to_num(7.0))
        rig.done([(slot, n)])
        at += n
