"""The per-row kernels of long steps (a norm a head with its gate, a gated norm a part) against 64 bits, at row counts on both
sides of every place where their dispatch changes, and a row's bits alone against those of the same row among many."""
import pytest
import torch

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
