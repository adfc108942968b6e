"""The kernels that take a projection apart for sink attention and latent attention have a form with 16-byte accesses and one an element
at a time; which one a step takes follows the rows' alignment alone, and both leave the same bits.  Rows an odd number of floats apart
take the second.  Queries are also held to the formula in 64 bits."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def step(T, P, gen):
    """Tokens of three requests at positions that lie apart, and their pages in any order."""
    pos = torch.randperm(6 * T, generator=gen, device=DEV)[:T].sort().values.to(torch.int32)
    req = torch.randint(0, 3, (T,), generator=gen, device=DEV, dtype=torch.int32)
    width = 6 * T // P + 1
    table = torch.randperm(3 * width, generator=gen, device=DEV).to(torch.int32).view(3, width)
    return SimpleNamespace(positions=pos, token_req=req, err=torch.zeros(1, dtype=torch.int32, device=DEV)), table


def both(rows, extra):
    """The same rows a multiple of four floats apart, and an odd number."""
    T, n = rows.shape
    for pad in (-n % 4 + extra, -n % 4 + 1):
        wide = torch.full((T, n + pad), float("nan"), device=DEV)
        wide[:, :n] = rows
        yield wide


@pytest.mark.parametrize("H,G,d,e,T", [(16, 4, 128, 128, 7), (3, 1, 20, 12, 300), (2, 2, 4, 4, 1), (33, 3, 128, 64, 5), (5, 5, 36, 132, 9)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("bias", [False, True])
def test_sink_attention_s_projection(H, G, d, e, T, dtype, bias):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(H * d + T)
    P, n = 8, H * d + G * (d + e) + H
    ctx, table = step(T, P, gen)
    rows = torch.randn(T, n, generator=gen, device=DEV)
    b = torch.randn(n - H, generator=gen, device=DEV) if bias else None
    got = []
    for proj in both(rows, 0):
        pages = torch.full((table.numel(), G, P, d + e), 7.0, dtype=dtype, device=DEV)
        got.append((*ops.sink_attn_prepare(proj, b, pages, ctx, table, H, G, d, e, 1e-5), pages))
    assert int(ctx.err.item()) == 0 and all(torch.equal(x, y) for x, y in zip(*got))
    sums = rows[:, :n - H].double() + (b.double() if bias else 0.0)
    step_of = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23        # one rounding (in bfloat16 of a float32 sum: twice)
    q, gate, pages = got[0]
    assert bool(((q.view(T, -1).double() - sums[:, :H * d]).abs() <= step_of * sums[:, :H * d].abs() + 1e-30).all())
    assert bool(((gate.double() - torch.sigmoid(rows[:, n - H:].double())).abs() <= 2.0 ** -21).all())
    page = table[ctx.token_req.long(), (ctx.positions // P).long()].long()
    kv = pages[page, :, (ctx.positions % P).long()].double()              # [T, G, d + e]
    k, v = sums[:, H * d:H * d + G * d].view(T, G, d), sums[:, H * d + G * d:].view(T, G, e)
    v = v * torch.rsqrt((v * v).mean(-1, keepdim=True) + 1e-5)
    assert bool(((kv[..., :d] - k).abs() <= step_of * k.abs() + 1e-30).all())
    assert bool(((kv[..., d:] - v).abs() <= (step_of + 2.0 ** -19) * v.abs() + 1e-30).all())


@pytest.mark.parametrize("H,d,rot,rank,rot_dims,halves", [
    (16, 128, 64, 512, 64, False), (33, 132, 4, 36, 4, False), (3, 20, 8, 64, 8, True),       # the rotation turns all of a part, four at a time
    (5, 36, 12, 60, 12, True),                                                                # halves of six: an element at a time
    (2, 8, 16, 32, 8, False), (2, 8, 16, 32, 8, True), (4, 4, 8, 30, 8, False),               # part of a part; rows of q_full off four
    (1, 4, 260, 8, 260, False)])                                                              # more angles than the table holds
@pytest.mark.parametrize("T", [5, 400])                                   # blocks of 1,024 threads and of 128
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_latent_attention_s_projection(H, d, rot, rank, rot_dims, halves, T, dtype):
    from ai_engine_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(H * d + T)
    P, n, dq = 16, H * (d + rot) + rank + rot, d + rot
    ctx, table = step(T, P, gen)
    rows = torch.randn(T, n, generator=gen, device=DEV)
    weight = torch.randn(rank, generator=gen, device=DEV)
    freq = 10000.0 ** (-torch.arange(rot_dims // 2, device=DEV) / (rot_dims // 2))
    short = torch.full((T,), -1, dtype=torch.int32, device=DEV)
    short[::3] = torch.arange(len(short[::3]), dtype=torch.int32, device=DEV)
    got = []
    for proj in both(rows, 4):
        outs = []
        for more in (dict(whole=True), dict(whole=True, short_row=short, n_short=len(short[::3])), dict(folded=False, whole=True)):
            pages = torch.full((table.numel(), 1, P, rank + rot), 7.0, dtype=dtype, device=DEV)
            plain, full, whole = ops.latent_prepare(proj, H, d, rot, rank, weight, 1e-5, freq, pages, ctx, table, dtype, True,
                                                    halves=halves, magnitude=1.25, **more)
            if full is not None:
                full = full[:, :, rank:]                                  # (the rest is another kernel's)
            if "short_row" in more:
                whole = whole[short < 0]
            outs += [t for t in (plain, full, whole, pages) if t is not None]
        got.append(outs)
    assert int(ctx.err.item()) == 0 and all(torch.equal(x, y) for x, y in zip(*got))
    plain, full, whole = got[0][:3]
    x = rows[:, :H * dq].view(T, H, dq)
    angle = (ctx.positions.float()[:, None] * freq).double()[:, None]     # (the product in float32, as the kernels make it)
    c, s, p, want = 1.25 * torch.cos(angle), 1.25 * torch.sin(angle), x[..., d:].double(), x[..., d:].double().clone()
    at = torch.arange(rot_dims // 2, device=DEV)
    i, j = (at, at + rot_dims // 2) if halves else (2 * at, 2 * at + 1)
    want[..., i], want[..., j] = p[..., i] * c - p[..., j] * s, p[..., j] * c + p[..., i] * s
    mag = p.abs().clone()
    mag[..., i] = mag[..., j] = 1.25 * (p[..., i].abs() + p[..., j].abs())
    assert torch.equal(plain, x[..., :d].to(dtype)) and torch.equal(whole[..., :d], x[..., :d].to(dtype))
    assert bool(((full.double() - want).abs() <= 2.0 ** -21 * mag).all())
    assert torch.equal(whole[..., d:], full.to(dtype))
