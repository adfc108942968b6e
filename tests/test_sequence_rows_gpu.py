"""The per-row kernels of long steps (a norm a head with its gate, a gated norm a part, the convolution over tiles of tokens)
against 64 bits, at row counts on both sides of every place where their dispatch changes, and a row's bits alone against those
of the same row among many."""
import pytest
import torch

from test_linear_recurrence_chunked_gpu import Ctx

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def close(got, ref, dtype, terms):
    """In units of 2^-24: a sum of positive terms behind one another in 32 lanes and five exchanges, halved by its root; an
    exponential of two units in the last place (four); twelve divisions, roots, products and sums.  bfloat16 rounds the result
    once on top."""
    bound = ((terms / 32 + 5) / 2 + 4 + 12) * 2.0 ** -24 + (0.0 if dtype == torch.float32 else 2.0 ** -8)
    assert bool(((got.double() - ref).abs() <= bound * ref.abs() + 1e-30).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dv", [32, 64, 128, 256, 96])
@pytest.mark.parametrize("T,H,gated,weighted", [(1, 3, True, True), (4095, 1, False, True), (1366, 3, True, False), (819, 5, True, True),
                                                (4096, 1, False, False)])
def test_norm_a_head_with_its_gate(T, H, gated, weighted, dv, dtype):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(T + dv)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    o, wide, w = rnd(T, H, dv), rnd(T, H * dv + 8), rnd(dv) if weighted else None
    g = wide[:, 4:4 + H * dv] if gated else None
    got = ops.head_norm_gate(o, g, w, 1e-5, dtype)
    ref = o.double() / torch.sqrt((o.double() ** 2).mean(-1, keepdim=True) + 1e-5)
    if weighted:
        ref = ref * w.double()
    if gated:
        ref = ref * torch.nn.functional.silu(g.double()).view(T, H, dv)
    close(got, ref.reshape(T, H * dv), dtype, dv)
    for t in {0, T // 2, T - 1}:
        assert torch.equal(ops.head_norm_gate(o[t:t + 1], g[t:t + 1] if gated else None, w, 1e-5, dtype)[0], got[t])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [128, 256, 512, 1024, 64])
@pytest.mark.parametrize("T,parts", [(1, 2), (1023, 1), (205, 5), (1025, 1)])
def test_gated_norm_a_part(T, parts, n, dtype):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(T + n)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    W = parts * n
    y, z, w = rnd(T, W), rnd(T, W + 12)[:, 8:8 + W], rnd(W)
    got = ops.gate_group_norm(y, z, w, parts, 1e-5, dtype)
    g = (y.double() * torch.nn.functional.silu(z.double())).view(T, parts, n)
    close(got, (g / torch.sqrt((g * g).mean(-1, keepdim=True) + 1e-5)).reshape(T, W) * w.double(), dtype, n)
    for t in {0, T // 2, T - 1}:
        assert torch.equal(ops.gate_group_norm(y[t:t + 1], z[t:t + 1], w, parts, 1e-5, dtype)[0], got[t])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("taps,residual,act,dup", [(2, True, None, 0), (3, False, "silu", 0), (4, False, "silu", 64), (4, True, None, 0)])
@pytest.mark.parametrize("lens", [[40, 1, 2, 17, 33], [300, 1, 1, 1], [16, 15, 3, 64], [1, 129]])
def test_convolution_over_tiles_of_tokens(taps, residual, act, dup, lens, dtype):
    """Tiles that begin inside a request and that hold several, portions shorter than the taps, lone tokens beside prompts: the
    outputs, the tail that each request keeps, and the bits of the kernel for short steps."""
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(taps + len(lens))
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    C, T = 192, sum(lens)
    assert T >= 8 * len(lens)                                     # the rule of the tiles
    wide, w, bias, tails = rnd(T, C + 8), rnd(C, taps), rnd(C), rnd(len(lens) + 1, taps - 1, C)
    u, slots = wide[:, 4:4 + C], list(range(len(lens)))[::-1]

    def step(rows, lens, slots, state):
        ctx = Ctx(lens, slots)
        ctx.token_req = torch.repeat_interleave(torch.arange(len(lens), dtype=torch.int32, device=DEV), torch.tensor(lens, device=DEV))
        out = ops.causal_conv(rows, w, bias, state, ctx, dtype, activation=act, residual=residual, dup_from=C - dup if dup else 0, dup_n=dup)
        assert int(ctx.err.item()) == 0
        return out

    state = tails.clone()
    got, at = step(u, lens, slots, state), 0
    for n, slot in zip(lens, slots):
        x = torch.cat([tails[slot], u[at:at + n]])
        assert torch.equal(state[slot], x[n:])
        terms = torch.stack([x[j:j + n].double() * w[:, j].double() for j in range(taps)] + ([u[at:at + n].double()] if residual else []))
        ref, mag = terms.sum(0) + bias.double(), terms.abs().sum(0) + bias.double().abs()
        if act:
            ref, mag = torch.nn.functional.silu(ref), 1.1 * mag   # its slope is at most 1.1
        ref, mag = (torch.cat([v, v[:, C - dup:]], dim=1) for v in (ref, mag))
        bound = (taps + 12) * 2.0 ** -24 * mag + (0.0 if dtype == torch.float32 else 2.0 ** -8) * ref.abs()
        assert bool(((got[at:at + n].double() - ref).abs() <= bound).all())
        one = tails.clone()                                       # seven tokens at a time: the kernel for short steps
        short = [step(u[at + i:at + min(i + 7, n)], [min(7, n - i)], [slot], one) for i in range(0, n, 7)]
        assert torch.equal(torch.cat(short), got[at:at + n]) and torch.equal(one[slot], state[slot])
        at += n
    assert torch.equal(state[len(lens)], tails[len(lens)])
