"""The gated delta rule that is parallel over chunks, against the recurrence in 64 bits and beside the kernel that walks a
request's chunks: both key sizes, value sizes at the edges of the blocks of columns, wide and narrow walks, portions at the edges
of chunks, a request that is not live, short portions and single tokens in the same step."""
import pytest
import torch

from test_linear_recurrence_chunked_gpu import DEV, Ctx

pytestmark = pytest.mark.gpu


def recurrence(q, k, v, beta, g, S, lens, slots):
    """q, k, v [T, H, .], beta, g [T, H], S [slots, H, d, e], float64: outputs and states."""
    out, S, at = torch.empty_like(v), S.clone(), 0
    for n, s in zip(lens, slots):
        for t in range(at, at + n):
            S[s] = S[s] * g[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.einsum("hde,hd->he", S[s], k[t]))
            S[s] = S[s] + k[t][:, :, None] * u[:, None, :]
            out[t] = torch.einsum("hde,hd->he", S[s], q[t])
        at += n
    return out, S


@pytest.mark.parametrize("H,G,d,e,lens,dead", [(2, 1, 128, 128, [64, 65], None), (3, 3, 64, 16, [300, 5, 1, 129, 32], None),
                                               (4, 2, 128, 48, [193, 40], 0), (40, 4, 64, 96, [130, 31], None),
                                               (20, 20, 128, 144, [63, 128, 1], None), (1, 1, 128, 80, [1025], None)])
def test_chunks_in_parallel(H, G, d, e, lens, dead, monkeypatch):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(d * 5 + e)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    T, slots = sum(lens), list(range(len(lens)))[::-1]
    rows = 1.5 * rnd(T, 2 * G * d + H * e)
    q, k, v = rows[:, :G * d], rows[:, G * d:2 * G * d], rows[:, 2 * G * d:]
    b_raw, a_raw, a_log, dt_bias = 2.0 * rnd(T, H + 1)[:, :H], 3.0 * rnd(T, H), 0.7 * rnd(H) - 0.5, 0.5 * rnd(H) - 1.0
    state0 = 0.5 * rnd(len(lens) + 1, H, d, e)
    ran = []
    inner = ops._delta_in_parallel
    monkeypatch.setattr(ops, "_delta_in_parallel", lambda *a: ran.append(inner(*a)) or ran[-1])

    def run(parallel):
        monkeypatch.setattr(ops, "DELTA_PARALLEL_CHUNKS", 1)
        monkeypatch.setattr(ops, "DELTA_PARALLEL_BYTES", 1 << 30 if parallel else 0)
        state, ctx = state0.clone(), Ctx(lens, slots)
        ctx.live = None if dead is None else torch.tensor([int(i != dead) for i in range(len(lens))], dtype=torch.int32, device=DEV)
        out = ops.delta_rule(q, k, v, b_raw, a_raw, a_log, dt_bias, d ** -0.5, 1e-6, state, ctx, H, G, d, e, chunked=True)
        assert int(ctx.err.item()) == 0
        return out, state

    out, state = run(True)
    assert ran == [True]
    other, other_state = run(False)
    assert ran == [True, False]
    heads = lambda t: t.double().reshape(T, G, d).repeat_interleave(H // G, dim=1)
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    g = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(a_raw.double() + dt_bias.double()))
    ref, S = recurrence(unit(heads(q)) * d ** -0.5, unit(heads(k)), v.double().reshape(T, H, e), torch.sigmoid(b_raw.double()), g,
                        state0.double(), lens, slots)
    if dead is not None:
        S[slots[dead]] = state0[slots[dead]].double()
    # pairs of bfloat16 values carry 2^-17 of each factor, a chunk adds up to 64 corrections: 2^-17 * sqrt(64) and a few factors
    for a, b, want in ((out, other, ref), (state, other_state, S)):
        for got in (a, b):
            assert float((got.double() - want).abs().max()) <= 3e-4 * float(want.std())
        rms = lambda got: float((got.double() - want).pow(2).mean().sqrt())
        assert rms(a) <= 1.1 * rms(b)                  # no less precise than chunk after chunk; 10 %: other sums' order
