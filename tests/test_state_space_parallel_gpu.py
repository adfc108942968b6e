"""The state-space recurrence that is parallel over chunks, against the recurrence in 64 bits on operands rounded to bfloat16
as the products see them, and beside the kernel that walks a request's chunks: odd states and heads, rows off the 16-byte
grid, portions at the edges of chunks, short portions and single tokens in the same step."""
import pytest
import torch

from test_linear_recurrence_chunked_gpu import DEV, Ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,hpg,N,dv,lens,pad", [(4, 2, 128, 64, [192, 5, 1, 64], 0), (2, 1, 64, 72, [300], 4), (6, 3, 100, 36, [33, 193, 31], 0),
                                                 (1, 1, 7, 130, [200, 32], 1), (3, 1, 16, 5, [257], 3), (2, 2, 36, 64, [63, 65, 448], 0),
                                                 (64, 8, 16, 8, [1280, 33], 0), (64, 2, 20, 12, [700], 0)])    # several heads a block
def test_chunks_in_parallel(H, hpg, N, dv, lens, pad, monkeypatch):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(N * 3 + dv)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    T, GN = sum(lens), H // hpg * N
    rows = rnd(T, H * dv + 2 * GN + pad)
    x, B, C = rows[:, :H * dv], rows[:, H * dv:H * dv + GN], rows[:, H * dv + GN:H * dv + 2 * GN]
    dt_raw, dt_bias, a_log, skip = 2.0 * rnd(T, H + 3)[:, :H], rnd(H), rnd(H) - 1.0, rnd(H)
    slots = list(range(len(lens)))[::-1]
    state0 = rnd(len(lens) + 1, H, N, dv)

    def run(parallel):
        monkeypatch.setattr(ops, "SSD_PARALLEL_TOKENS", 32 if parallel else 1 << 30)
        state, ctx = state0.clone(), Ctx(lens, slots)
        out = ops.linear_recurrence(C, B, x, None, None, 1.0, 1.0, state, ctx, H, N, dv, heads_per_group=hpg, dt_raw=dt_raw,
                                    dt_bias=dt_bias, a_log=a_log, skip=skip, chunked=True)
        assert int(ctx.err.item()) == 0
        return out, state

    entered, real = [], ops.library
    monkeypatch.setattr(ops, "library", lambda name: entered.append(name) or real(name))
    out, state = run(True)
    assert "state_space_parallel.cu" in entered and "state_space_chunked.cu" not in entered
    other, other_state = run(False)
    assert entered.count("state_space_parallel.cu") == 1 and "state_space_chunked.cu" in entered
    rounded = lambda t, n: t.to(torch.bfloat16).double().reshape(T, n, -1).repeat_interleave(H // n, dim=1)
    dt = torch.nn.functional.softplus(dt_raw.double() + dt_bias.double())
    a = torch.exp(-torch.exp(a_log.double()) * dt)
    ref, S, mag, M, at = torch.empty(T, H, dv, device=DEV, dtype=torch.float64), state0.double(), None, state0.double().abs(), 0
    mag = torch.empty_like(ref)
    full = lambda t, n: t.double().reshape(T, n, -1).repeat_interleave(H // n, dim=1)
    for n, s in zip(lens, slots):
        pick = rounded if n >= ops.SSD_MIN_TOKENS else full       # shorter portions take the token-by-token kernel
        xs, Bs, Cs = pick(x, H), pick(B, H // hpg), pick(C, H // hpg)
        for t in range(at, at + n):
            S[s] = S[s] * a[t][:, None, None] + Bs[t][:, :, None] * (xs[t] * dt[t][:, None])[:, None, :]
            M[s] = M[s] * a[t][:, None, None] + Bs[t].abs()[:, :, None] * (xs[t].abs() * dt[t][:, None])[:, None, :]
            ref[t] = torch.einsum("hnd,hn->hd", S[s], Cs[t]) + skip.double()[:, None] * xs[t]
            mag[t] = torch.einsum("hnd,hn->hd", M[s], Cs[t].abs()) + (skip.double()[:, None] * xs[t]).abs()
        at += n
    # pairs of bfloat16 values carry 2^-17; decays' exponents (sums of 64 steps, up to some tens) 2^-24 times their size
    for got, want, size in ((out, ref, mag), (state, S, M), (other, ref, mag), (other_state, S, M)):
        assert bool(((got.double() - want).abs() <= 2.0 ** -14 * size + 1e-30).all())
