"""The chunk-parallel linear recurrence against the recurrence in 64 bits: sizes at the edges of its tiles, portions at the
edges of its chunks, the three forms of the decay, decays of 0 and 1, requests short enough for the token-by-token kernel
beside long ones, states carried from step to step."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


class Ctx:
    def __init__(self, lens, slots):
        starts = np.concatenate([[0], np.cumsum(lens)[:-1]])
        i32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device=DEV)
        self.q_start, self.q_len, self.slots = i32(starts), i32(lens), i32(slots)
        self.h_q_len, self.R, self.max_q_len = np.asarray(lens), len(lens), max(lens)
        self.err = torch.zeros(1, dtype=torch.int32, device=DEV)


def reference(q, k, v, a, S, lens, slots):
    """q, k, a [T, H, d], v [T, H, e], S [slots, H, d, e], all float64: outputs and states."""
    out, S, at = torch.empty_like(v), S.clone(), 0
    for n, s in zip(lens, slots):
        for t in range(at, at + n):
            S[s] = S[s] * a[t][:, :, None] + k[t][:, :, None] * v[t][:, None, :]
            out[t] = torch.einsum("hde,hd->he", S[s], q[t])
        at += n
    return out, S


@pytest.mark.parametrize("form", ["token", "head", "keyless"])
@pytest.mark.parametrize("H,d,e,lens", [(2, 128, 128, [64]), (1, 128, 128, [300, 5, 128, 7, 8]), (3, 64, 64, [65, 129]),
                                        (2, 60, 68, [127, 9, 1]), (1, 4, 128, [191]), (2, 68, 4, [200, 64, 70])])
def test_chunks_against_the_recurrence(form, H, d, e, lens, monkeypatch):
    from ai_engine_b200.kernels import ops
    monkeypatch.setattr(ops, "LC_MIN_WORK", 0)              # small steps too
    taken, real = [], ops._recurrence_in_chunks
    monkeypatch.setattr(ops, "_recurrence_in_chunks", lambda *a: taken.append(real(*a)) or taken[-1])
    gen = torch.Generator(device=DEV).manual_seed(d * 7 + e + len(lens))
    T, slots = sum(lens), list(range(len(lens)))[::-1]
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    rows = rnd(T, 2 * H * d + H * e + 4)                    # one product's output: q | k | v | something else
    q, k, v = rows[:, :H * d], rows[:, H * d:2 * H * d], rows[:, 2 * H * d:2 * H * d + H * e]
    state0 = rnd(len(lens) + 1, H, d, e)
    scale, lower, bias, decay_tok, decay_head = 0.3, None, None, None, None
    q64, k64, v64 = (t.double().reshape(T, H, -1) for t in (q, k, v))
    if form == "keyless":
        lower, bias, decay_tok = torch.rand(H * d, generator=gen, device=DEV), rnd(H * d), 3.0 * rnd(T, H * d)
        lower[: H * d // 4] = 0.0
        # the gate in float32, as the kernels make it: 64 bits of its logits would differ by its own rounding
        f = lower + (1.0 - lower) * (1.0 / (1.0 + torch.exp(-(decay_tok + bias))))
        a64, k64 = f.double().view(T, H, d), (1.0 - f.double()).view(T, H, d)
        q64, scale = torch.nn.functional.silu(q64), 1.0
    elif form == "token":
        decay_tok = torch.sigmoid(4.0 * rnd(T, H * d + 4))[:, :H * d]
        decay_tok[::7, ::5], decay_tok[3::11, 1::3] = 0.0, 1.0
        a64, q64 = decay_tok.double().reshape(T, H, d), q64 * scale
    else:
        decay_head = torch.linspace(0.2, 0.999, H, device=DEV)
        a64, q64 = decay_head.double()[None, :, None].expand(T, H, d), q64 * scale
    ctx, state = Ctx(lens, slots), state0.clone()
    out = ops.linear_recurrence(q, None if form == "keyless" else k, v, decay_tok, decay_head, scale, 1.0, state, ctx, H, d, e,
                                forget_lower=lower, forget_bias=bias)
    assert taken == [ops.LC_MIN_TOKENS]
    ref, ref_state = reference(q64, k64, v64, a64, state0.double(), lens, slots)
    mag, mag_state = reference(q64.abs(), k64.abs(), v64.abs(), a64, state0.double().abs(), lens, slots)
    # every term is rounded once per factor and addition that it passes: at most two a token of its chunk, a chunk of its
    # request and a channel; eight more for the gate and its exponential
    steps = 2 * 64 + max(lens) // 32 + d + 8
    assert bool(((out.double() - ref).abs() <= steps * 2.0 ** -24 * mag + 1e-30).all())
    assert bool(((state.double() - ref_state).abs() <= steps * 2.0 ** -24 * mag_state + 1e-30).all())
    assert torch.equal(state[len(lens)], state0[len(lens)]) and int(ctx.err.item()) == 0


def test_strides_and_addresses_that_are_not_taken_go_the_general_way():
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(5)
    T, H, d = 130, 2, 8
    rows = torch.randn(T, 3 * H * d + 1, generator=gen, device=DEV)           # an odd row stride
    for at in (0, 1):
        q, k, v = (rows[:, at + i * H * d:at + (i + 1) * H * d] for i in range(3))
        whole = [t.contiguous() for t in (q, k, v)]
        dec, outs = torch.full((H,), 0.9, device=DEV), []
        for a, b, c in ((q, k, v), whole):
            state = torch.zeros(1, H, d, d, device=DEV)
            outs.append((ops.linear_recurrence(a, b, c, None, dec, 1.0, 1.0, state, Ctx([T], [0]), H, d, d), state))
        for x, y in zip(*outs):
            assert float((x - y).abs().max()) < 1e-5 * float(y.abs().max())


def test_a_slot_outside_its_table_is_flagged_and_writes_no_state():
    from ai_engine_b200.kernels import ops
    x = torch.randn(128, 24, device=DEV)
    state = torch.ones(1, 1, 8, 8, device=DEV)
    ctx = Ctx([128], [1])
    ops.linear_recurrence(x[:, :8], x[:, 8:16], x[:, 16:], None, torch.ones(1, device=DEV), 1.0, 1.0, state, ctx, 1, 8, 8)
    assert int(ctx.err.item()) == 8 and bool((state == 1).all())


@pytest.mark.parametrize("what", ["k", "v", "q", "decay"])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_a_value_that_is_not_finite_reaches_no_earlier_token(what, value):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(9)
    T, H, d = 200, 2, 64
    rows, clean = torch.randn(T, 4 * H * d, generator=gen, device=DEV), None
    rows[:, 3 * H * d:] = torch.sigmoid(rows[:, 3 * H * d:])
    for at in (None, 5, 64, 77, 126, 199):
        x = rows.clone()
        if at is not None:
            x[at, "qkv".find(what) * H * d if what != "decay" else 3 * H * d:][:H * d] = value
        q, k, v, a = (x[:, i * H * d:(i + 1) * H * d] for i in range(4))
        out = ops.linear_recurrence(q, k, v, a, None, 1.0, 1.0, torch.zeros(1, H, d, d, device=DEV), Ctx([T], [0]), H, d, d)
        if at is None:
            clean = out
        else:
            assert torch.equal(out[:at], clean[:at]) and not bool(torch.isfinite(out[at]).all())
