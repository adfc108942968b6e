"""Which kernel takes a portion is decided by the portion, never by what else is in the step: the state that a request leaves has
the same bits alone and beside others, its outputs up to the order of the token-by-token kernel's sum over a state's rows, which
follows the step's shape.  The float32 engine walks a recurrence token by token, so there the state's bits do not depend on how
a prompt was cut either."""
import pytest
import torch

from test_linear_recurrence_chunked_gpu import DEV, Ctx
from test_pifutar_parts_gpu import linear_part
from zupitar_helpers import Rig, load

pytestmark = pytest.mark.gpu


def alone_and_beside(run, lens, exact):
    """run([(request, tokens)]): (outputs, state) of every request of one step.  exact(n): the outputs' bits are the same too.
    (A step of single tokens may have a kernel of its own.)"""
    together = run(list(enumerate(lens)))
    near = lambda a, b: float((a - b).abs().max()) <= 1e-5 * float(a.abs().max())
    for i, n in enumerate(lens):
        (out, state), (out2, state2) = run([(i, n)])[0], together[i]
        assert torch.equal(state, state2) if n > 1 else near(state, state2), (i, n)
        assert torch.equal(out, out2) if exact(n) else near(out, out2), (i, n)


def linear(H, lens, keyless):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(H)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    d = 32
    rows = [rnd(n, 4 * H * d) for n in lens]
    states, lower = rnd(len(lens), H, d, d), torch.rand(H * d, generator=gen, device=DEV)

    def run(reqs):
        x, state = torch.cat([rows[i] for i, _ in reqs]), states.clone()
        q, k, v, a = (x[:, j * H * d:(j + 1) * H * d] for j in range(4))
        ctx = Ctx([n for _, n in reqs], [i for i, _ in reqs])
        out = ops.linear_recurrence(q, None if keyless else k, v, a if keyless else torch.sigmoid(a), None, 0.3, 1.0, state, ctx, H, d, d,
                                    forget_lower=lower if keyless else None)
        assert int(ctx.err.item()) == 0
        return [(o, state[i]) for o, (i, _) in zip(out.split([n for _, n in reqs]), reqs)]

    return run


@pytest.mark.parametrize("keyless", [False, True])
@pytest.mark.parametrize("H,lens", [(16, [40, 300, 1, 53, 54, 9]), (40, [41, 12, 43, 42]),
                                    (16, [1] * 33 + [70] + [3] * 34 + [130, 64])])
def test_linear_recurrence(H, lens, keyless):
    from ai_engine_b200.kernels import ops
    alone_and_beside(linear(H, lens, keyless), lens, lambda n: n >= ops.lc_min_len(H))


@pytest.mark.parametrize("kind,extra", [("retention", [0.5, 0.9, 0.99]), ("gla", 8.0)])
def test_float32_linear_attention_whole_and_in_portions(kind, extra):
    D, H, d, dv, n = 48, 3, 16, 32, 190
    g = torch.Generator().manual_seed(5)
    r = lambda *s: torch.randn(*s, generator=g) / s[-1] ** 0.5
    ts = {"q": r(H * d, D), "k": r(H * d, D), "v": r(H * dv, D), "g": r(H * dv, D), "o": r(D, H * dv)}
    ts.update({"norm": 1.0 + r(dv), "a1": r(6, D), "a2": r(H * d, 6), "a2.b": 2.0 + r(H * d)} if kind == "gla" else {})
    part = load(linear_part(torch.float32, D, kind, H, d, dv, extra), ts, torch.float32)
    h, outs, states = torch.randn(n, D, generator=g), [], []
    for cuts in ([n], [120, 7, 1, 62]):
        rig, at, got = Rig(part, torch.float32), 0, []
        slot = rig.admit()
        for c in cuts:
            ctx, lc = rig.step([(slot, c)])
            got.append(part.forward(h[at:at + c].to(DEV), ctx, lc))
            rig.done([(slot, c)])
            at += c
        outs.append(torch.cat([o.sum(0) if o.dim() == 3 else o for o in got]))
        states.append(lc.state[slot].clone())
    assert torch.equal(*states)
    assert float((outs[0] - outs[1]).abs().max()) <= 1e-5 * float(outs[0].abs().max())


def state_space(H, hpg, lens):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(H)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    N, dv, G = 32, 32, H // hpg
    rows, steps = [rnd(n, H * dv + 2 * G * N) for n in lens], [rnd(n, H) for n in lens]
    states, bias, a_log, skip = rnd(len(lens), H, N, dv), rnd(H), rnd(H) - 1.0, rnd(H)

    def run(reqs):
        x, dt, state = torch.cat([rows[i] for i, _ in reqs]), torch.cat([steps[i] for i, _ in reqs]), states.clone()
        ctx = Ctx([n for _, n in reqs], [i for i, _ in reqs])
        out = ops.linear_recurrence(x[:, H * dv + G * N:], x[:, H * dv:H * dv + G * N], x[:, :H * dv], None, None, 1.0, 1.0, state, ctx,
                                    H, N, dv, heads_per_group=hpg, dt_raw=dt, dt_bias=bias, a_log=a_log, skip=skip, chunked=True)
        assert int(ctx.err.item()) == 0
        return [(o, state[i]) for o, (i, _) in zip(out.split([n for _, n in reqs]), reqs)]

    return run


@pytest.mark.parametrize("H,hpg,lens", [(4, 2, [159, 40, 160, 5, 300, 1, 64]), (32, 4, [31, 32, 130, 100]),
                                        (4, 1, [1] * 33 + [170] + [3] * 34 + [230, 40])])
def test_state_space(H, hpg, lens):
    from ai_engine_b200.kernels import ops
    alone_and_beside(state_space(H, hpg, lens), lens, lambda n: n >= ops.SSD_MIN_TOKENS)


def delta(H, G, lens):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(H)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    d, e = 64, 32
    rows, gates = [rnd(n, 2 * G * d + H * e) for n in lens], [rnd(n, 2 * H) for n in lens]
    states, a_log, bias = rnd(len(lens), H, d, e), rnd(H) - 1.0, rnd(H)

    def run(reqs):
        x, g, state = torch.cat([rows[i] for i, _ in reqs]), torch.cat([gates[i] for i, _ in reqs]), states.clone()
        ctx = Ctx([n for _, n in reqs], [i for i, _ in reqs])
        ctx.live = None
        out = ops.delta_rule(x[:, :G * d], x[:, G * d:2 * G * d], x[:, 2 * G * d:], g[:, :H], g[:, H:], a_log, bias, d ** -0.5, 1e-6,
                             state, ctx, H, G, d, e, chunked=True)
        assert int(ctx.err.item()) == 0
        return [(o, state[i]) for o, (i, _) in zip(out.split([n for _, n in reqs]), reqs)]

    return run


@pytest.mark.parametrize("H,G,lens", [(4, 2, [192, 40, 193, 5, 300, 1, 64]), (24, 24, [31, 32, 130, 100, 280]),
                                      (2, 1, [1] * 33 + [200] + [3] * 34 + [257, 40])])
def test_delta_rule(H, G, lens):
    alone_and_beside(delta(H, G, lens), lens, lambda n: n > 1)


def test_a_prompt_beside_so_many_lone_tokens_that_a_grid_over_all_of_them_would_be_too_large(monkeypatch):
    from ai_engine_b200.kernels import ops
    taken, real = [], ops._recurrence_in_chunks
    monkeypatch.setattr(ops, "_recurrence_in_chunks", lambda *a: taken.append(real(*a)) or taken[-1])
    H, d, lens = 64, 4, [1] * 1100 + [40]
    x = torch.randn(sum(lens), 3 * H * d, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV)
    decay = torch.full((H,), 0.9, device=DEV)

    def run(rows, lens):
        state, ctx = torch.zeros(len(lens), H, d, d, device=DEV), Ctx(lens, list(range(len(lens))))
        q, k, v = (rows[:, i * H * d:(i + 1) * H * d] for i in range(3))
        out = ops.linear_recurrence(q, k, v, None, decay, 1.0, 1.0, state, ctx, H, d, d)
        assert int(ctx.err.item()) == 0
        return out[-40:], state[-1]

    for a, b in zip(run(x, lens), run(x[-40:], [40])):
        assert torch.equal(a, b)
    assert taken == [ops.lc_min_len(H)] * 2


@pytest.mark.parametrize("make,sizes,lens,head_bytes", [
    (linear, (6, False), [300, 1, 130, 200, 64, 190], 4 * 32 * 32), (state_space, (6, 3), [300, 1, 165, 40, 513, 200], 4 * 32 * 32),
    (delta, (6, 2), [300, 1, 200, 40, 513, 200], 64 * (8 * 64 + 4 * 32) + 4 * 64 * 32 + 4)])
def test_scratch_has_a_bound_and_no_bit_depends_on_it(make, sizes, lens, head_bytes, monkeypatch):
    from ai_engine_b200.kernels import ops
    reqs = list(enumerate(lens))
    run = make(*sizes[:1], lens, sizes[1]) if make is linear else make(*sizes, lens)
    want, sizes_asked, real = run(reqs), [], torch.empty
    for budget in (40 * head_bytes, 10 * head_bytes, 1):          # some portions together, heads apart, one head at a time
        for name in ("CHUNK_STATES_BYTES", "DELTA_PARALLEL_BYTES"):
            monkeypatch.setattr(ops, name, budget)
        with monkeypatch.context() as m:
            m.setattr(ops, "_scratch", lambda device, *sizes, f=ops._scratch: sizes_asked.append(sum(sizes)) or f(device, *sizes))
            got = run(reqs)
        longest = max(-(-n // 64) for n in lens)
        assert sizes_asked.pop() <= 1.04 * max(budget, longest * head_bytes) and not sizes_asked      # 4 %: what the decays take
        for (a, b), (c, d) in zip(want, got):
            assert torch.equal(a, c) and torch.equal(b, d)
    monkeypatch.undo()

    def full(shape, *a, **k):
        raise torch.OutOfMemoryError("no room")

    with monkeypatch.context() as m:                              # no room at all: a kernel that needs none
        m.setattr(ops, "_scratch", lambda device, *sizes, f=ops._scratch: [m.setattr(torch, "empty", full), f(device, *sizes),
                                                                          m.setattr(torch, "empty", real)][1])
        got = run(reqs)
    for (a, b), (c, d) in zip(want, got):
        assert float((a - c).abs().max()) <= 2e-3 * float(a.abs().max()) and float((b - d).abs().max()) <= 2e-3 * float(b.abs().max())
