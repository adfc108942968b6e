"""The work that is measured: single layers, blocks and decode steps of the architectures this engine serves, at the
sizes of `bench.py`'s shapes, each through the entry points a program calls.

Three ways in:

* `step`: `StepRunner.step` of a whole model (decode steps, replayed from a captured graph as the engine does), which
  returns logits;
* `block`: one layer's `block.forward` on the residual stream, closed by the model's final norm;
* one part's `forward` (a mixer or a feed-forward) on a real cache and step context, for each family of layers.

A case names its requests as text, "cached+new,cached+new,...": tokens that are in the cache already and tokens the
step brings.  `cuts` feeds every request's new tokens in that many portions, one step behind the other, as a long prompt
is fed under a token budget.
"""
import math

import torch

import ai_engine_b200 as aie
from ai_engine_b200.cache import PagedCache
from ai_engine_b200.engine.step import StepContext, StepEntry, StepRunner
from ai_engine_b200.parts import BuildEnv, CacheNeed, Model, PartSpec, lookup
from ai_engine_b200.weights.loader import from_tensors

DEV = "cuda:0"
PAGE = 16
EPS = 1e-5
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}

# Layer sizes of the Llama shapes that bench.py runs.
LLAMA_8B = dict(hidden=4096, inter=14336, heads=32, kv_heads=8, head_dim=128, theta=500000.0)
LLAMA_3B = dict(hidden=3072, inter=8192, heads=24, kv_heads=8, head_dim=128, theta=500000.0)
LLAMA_1B = dict(hidden=2048, inter=8192, heads=32, kv_heads=8, head_dim=64, theta=500000.0)


def _ragged(lo, hi, n, new):
    """n requests with cached lengths spread over lo .. hi (not in order) that bring `new` tokens each."""
    return ",".join(f"{lo + (hi - lo) * ((i * 37) % n) // max(1, n - 1)}+{new}" for i in range(n))


def _latent(width, **more):
    return dict(kind="latent", hidden=width, heads=width // 128, head_dim=128, rot=64, value_dim=128,
                rank=min(512, max(256, width // 4)), window=0, sink=False, exact_weights=False, cuts=1, **more)


def _sink(width, **more):
    return dict(kind="sink", hidden=width, heads=width // 128, kv_heads=max(1, width // 512), head_dim=128, value_dim=128,
                window=1024, keep_first=4, cuts=1, **more)


def _linear(kind, width, **more):
    return dict(kind=kind, hidden=width, heads=width // 128, head_dim=128, value_dim=128, **more)


def _ssm(width, **more):
    return dict(kind="ssm", hidden=width, heads=width // 32, value_dim=64, state=128, groups=8, taps=4, norm_groups=8, **more)


def _moe(width, tokens):
    return dict(kind="moe", hidden=width, experts=32, top=4, inter=width // 2, groups=4, keep=2, shared=width,
                requests=f"0+{tokens}", cuts=1)


def listed():
    return [
        # one user's decoded token on a small model: latency, a chain of small kernels
        dict(name="decode_one", kind="step", dtype="bf16", layers=8, vocab=128256, requests="1023+1", **LLAMA_1B),
        # a serving step: 64 requests of mixed context lengths
        dict(name="decode_many", kind="step", dtype="bf16", layers=4, vocab=128256, requests=_ragged(128, 4096, 64, 1), **LLAMA_8B),
        # a prompt step of the serving loop: a whole prompt, a later portion of another, and decoded tokens beside them
        dict(name="prompt_block", kind="block", dtype="bf16",
             requests="0+1531,700+500," + _ragged(200, 2000, 17, 1), **LLAMA_8B),
        # the 32-bit path, which results are checked with: an odd prompt beside a later portion of another
        dict(name="prompt_block_fp32", kind="block", dtype="fp32", requests="0+384,100+129", **LLAMA_1B),
        # gated linear attention over one prompt of a full step
        _linear("gla", 2048, name="gla_prompt", requests="0+2048", cuts=1),
        # keyless linear attention (a forget gate) over ragged prompts, each in two portions
        _linear("hgrn", 2048, name="hgrn_prompts", requests="0+1237,0+700,0+111", cuts=2),
        # attention over a compressed cache, a prompt's later portion under a window
        dict(_latent(2048, name="latent_prompt", requests="1024+2048"), window=1024),
        # the same without a window, decoding for 64 requests
        _latent(2048, name="latent_decode", requests=_ragged(512, 4096, 64, 1)),
        # windowed attention with distance bias, kept first tokens, a sink and gates; a later portion and a new prompt
        _sink(2048, name="sink_prompt", requests="1000+1900,0+148"),
        # the gated delta rule over a prompt in two portions
        _linear("delta", 2048, name="delta_prompt", requests="0+2048", cuts=2, qk_heads=8, taps=4),
        # a state-space layer over two prompts
        _ssm(2048, name="ssm_prompts", requests="0+1500,0+548", cuts=1),
        # routed experts beside a shared one, an odd number of tokens
        dict(_moe(2048, 1711), name="experts_prompt"),
    ]


def draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["step", "block", "block_fp32", "gla", "hgrn", "latent", "latent_decode", "sink", "delta", "ssm", "moe"])
    width = rng.choice([1024, 2048])

    def prompts(most, cached):
        n = rng.randint(1, 4)
        return ",".join(f"{rng.randint(1, cached) if cached and rng.random() < 0.5 else 0}+{log(200, most) // n + rng.randint(0, 9)}"
                        for _ in range(n))

    if kind == "step":
        n = log(1, 64)
        lo = rng.randint(1, 1500)
        return dict(kind="step", dtype="bf16", layers=rng.randint(1, 3), vocab=rng.choice([32000, 128256]),
                    requests=_ragged(lo, lo + rng.randint(0, 2500), n, 1), **rng.choice([LLAMA_8B, LLAMA_3B, LLAMA_1B]))
    if kind == "block":
        return dict(kind="block", dtype="bf16", requests=prompts(2000, 3000), **rng.choice([LLAMA_8B, LLAMA_3B, LLAMA_1B]))
    if kind == "block_fp32":
        return dict(kind="block", dtype="fp32", requests=prompts(500, 300), **LLAMA_1B)
    if kind in ("gla", "hgrn"):
        return _linear(kind, width, requests=prompts(4000, 0), cuts=rng.randint(1, 2))
    if kind == "delta":
        return _linear("delta", width, requests=prompts(3000, 0), cuts=rng.randint(1, 2), qk_heads=width // 256, taps=4)
    if kind == "ssm":
        return _ssm(width, requests=prompts(3000, 0), cuts=rng.randint(1, 2))
    if kind == "latent":
        c = _latent(width, requests=prompts(2500, 3000))
        c.update(window=rng.choice([0, 1024]), sink=rng.random() < 0.5, exact_weights=rng.random() < 0.5)
        return c
    if kind == "latent_decode":
        lo = rng.randint(1, 2000)
        return _latent(width, requests=_ragged(lo, lo + rng.randint(0, 3000), log(2, 64), 1))
    if kind == "sink":
        return _sink(width, requests=prompts(2500, 3000))
    return _moe(width, log(70, 3000))


# ---------------------------------------------------------------------------------------------------
# inputs, from the seed alone
def _requests(case):
    return [tuple(int(v) for v in r.split("+")) for r in case["requests"].split(",")]


def _portions(case):
    """For every step the list of (request, cached before it, tokens)."""
    cuts, steps = case.get("cuts", 1), []
    for k in range(cuts):
        rows = [(i, c + n * k // cuts, n * (k + 1) // cuts - n * k // cuts) for i, (c, n) in enumerate(_requests(case))]
        steps.append([r for r in rows if r[2]])
    return steps


def _first_pages(case):
    """First page of every request (pages of a request follow one another) and the number of pages."""
    out, at = [], 0
    for c, n in _requests(case):
        out.append(at)
        at += -(-(c + n) // PAGE)
    return out, at


def _llama_weights(case, rnd, layers, vocab):
    D, F, H, K, d = (case[k] for k in ("hidden", "inter", "heads", "kv_heads", "head_dim"))
    w = {"model.embed_tokens.weight": rnd(vocab, D), "model.norm.weight": rnd(D, std=0.1, mean=1.0),
         "lm_head.weight": rnd(vocab, D, std=D ** -0.5)}
    for i in range(layers):
        p = f"model.layers.{i}."
        w[p + "input_layernorm.weight"] = rnd(D, std=0.1, mean=1.0)
        w[p + "post_attention_layernorm.weight"] = rnd(D, std=0.1, mean=1.0)
        for name, shape in (("self_attn.q_proj", (H * d, D)), ("self_attn.k_proj", (K * d, D)), ("self_attn.v_proj", (K * d, D)),
                            ("self_attn.o_proj", (D, H * d)), ("mlp.gate_proj", (F, D)), ("mlp.up_proj", (F, D)),
                            ("mlp.down_proj", (D, F))):
            w[p + name + ".weight"] = rnd(*shape, std=shape[1] ** -0.5)
    return w


def _weights(case, rnd):
    k, D = case["kind"], case["hidden"]
    lin = lambda n, m: rnd(n, m, std=m ** -0.5)
    if k == "step":
        return _llama_weights(case, rnd, case["layers"], case["vocab"])
    if k == "block":
        return _llama_weights(case, rnd, 1, 64)
    if k == "moe":
        E, F, Fs = case["experts"], case["inter"], case["shared"]
        w = {"router": rnd(E, D, std=2.0 * D ** -0.5)}
        for e in range(E):
            w.update({f"e{e}.gate": lin(F, D), f"e{e}.up": lin(F, D), f"e{e}.down": lin(D, F)})
        return dict(w, **{"s.gate": lin(Fs, D), "s.up": lin(Fs, D), "s.down": lin(D, Fs)})
    H = case["heads"]
    if k == "ssm":
        inner, N, G, t = H * case["value_dim"], case["state"], case["groups"], case["taps"]
        return {"in": lin(2 * inner + 2 * G * N + H, D), "conv": rnd(inner + 2 * G * N, t, std=0.4),
                "conv_bias": rnd(inner + 2 * G * N, std=0.1), "dt_bias": rnd(H, mean=-1.0, std=0.5),
                "a_log": rnd(H, mean=-0.5, std=0.5), "skip": rnd(H, mean=1.0, std=0.2),
                "norm": rnd(inner, mean=1.0, std=0.1), "o": lin(D, inner)}
    d, e = case["head_dim"], case["value_dim"]
    if k == "gla":
        return {"q": lin(H * d, D), "k": lin(H * d, D), "v": lin(H * e, D), "g": lin(H * e, D), "o": lin(D, H * e),
                "a1": lin(16, D), "a2": lin(H * d, 16), "a2_bias": rnd(H * d, mean=3.0, std=1.0)}
    if k == "hgrn":
        return {"q": lin(H * d, D), "f": lin(H * d, D), "v": lin(H * e, D), "o": lin(D, H * e),
                "f_bias": rnd(H * d, mean=1.0, std=1.0), "lower": rnd(H * d, mean=0.3, std=0.1).clamp(0.0, 0.95),
                "norm": rnd(e, mean=1.0, std=0.1)}
    if k == "latent":
        rank, rot = case["rank"], case["rot"]
        w = {"q": lin(H * (d + rot), D), "dkv": lin(rank + rot, D), "dkv_norm": rnd(rank, mean=1.0, std=0.1),
             "uk": lin(H * d, rank), "uv": lin(H * e, rank), "o": lin(D, H * e)}
        return dict(w, sink=rnd(H)) if case["sink"] else w
    if k == "sink":
        G = case["kv_heads"]
        return {"q": lin(H * d, D), "k": lin(G * d, D), "v": lin(G * e, D), "o": lin(D, H * e), "g": lin(H, D),
                "q_bias": rnd(H * d, std=0.1), "k_bias": rnd(G * d, std=0.1), "v_bias": rnd(G * e, std=0.1),
                "temp": rnd(H, mean=1.0, std=0.2), "sink": rnd(H)}
    G, t = case["qk_heads"], case["taps"]                                      # delta
    return {"q": lin(G * d, D), "k": lin(G * d, D), "v": lin(H * e, D), "g": lin(H * e, D), "b": lin(H, D), "a": lin(H, D),
            "q_conv": rnd(G * d, t, std=0.4), "k_conv": rnd(G * d, t, std=0.4), "v_conv": rnd(H * e, t, std=0.4),
            "a_log": rnd(H, mean=-0.5, std=0.5), "dt_bias": rnd(H, mean=-1.0, std=0.5), "norm": rnd(e, mean=1.0, std=0.1),
            "o": lin(D, H * e)}


def _pool_shape(case):
    """[runs, planes, kv heads, row] of the paged cache, None without one."""
    k = case["kind"]
    if k in ("step", "block"):
        return case.get("layers", 1), 2, case["kv_heads"], case["head_dim"]
    if k == "latent":
        return 1, 1, 1, case["rank"] + case["rot"]
    if k == "sink":
        return 1, 1, case["kv_heads"], case["head_dim"] + case["value_dim"]
    return None


def _inputs(case, seed):
    """(weights by name, rows per request [tokens, hidden] or token ids, cache pool, residual rows that a branch joins)."""
    gen = torch.Generator(device=DEV).manual_seed(1000003 * seed + 17)

    def rnd(*shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
        return torch.empty(shape, device=DEV).normal_(mean, std, generator=gen).to(dtype)

    w = _weights(case, rnd)
    reqs, D = _requests(case), case["hidden"]
    if case["kind"] == "step":
        rows = [torch.randint(0, case["vocab"], (n,), generator=gen, device=DEV) for _, n in reqs]
    else:
        # what a norm hands to a mixer; a block gets a residual stream in float32
        rows = [rnd(n, D, dtype=torch.float32 if case["kind"] == "block" else torch.bfloat16) for _, n in reqs]
    pool = None
    if _pool_shape(case):
        runs, planes, K, row = _pool_shape(case)
        pool = rnd(runs, planes, _first_pages(case)[1], K, PAGE, row, dtype=DTYPES[case.get("dtype", "bf16")])
    return w, rows, pool, rnd(len(reqs), D, dtype=torch.float32)


def _spec(case):
    k, D = case["kind"], case["hidden"]
    name = lambda *ns: {n: n for n in ns}
    if k == "moe":
        return "feed_forward", PartSpec("routed_moe", dict(
            hidden_size=D, num_experts=case["experts"], top=case["top"], intermediate_size=case["inter"], groups=case["groups"],
            keep=case["keep"], score="sigmoid", group_top=2, normalise=True, route_scale=2.0,
            shared_intermediate_size=case["shared"]),
            dict(router="router", gate="e{e}.gate", up="e{e}.up", down="e{e}.down", shared_gate="s.gate", shared_up="s.up",
                 shared_down="s.down"))
    if k == "ssm":
        return "mixer", PartSpec("scalar_decay_state_space", dict(
            hidden_size=D, num_heads=case["heads"], value_dim=case["value_dim"], state_size=case["state"], groups=case["groups"],
            taps=case["taps"], norm_groups=case["norm_groups"], eps=EPS),
            name("in", "conv", "conv_bias", "dt_bias", "a_log", "skip", "norm", "o"))
    sizes = dict(hidden_size=D, num_heads=case["heads"], eps=EPS)
    if k == "latent":
        return "mixer", PartSpec("latent_attention", dict(
            sizes, head_dim=case["head_dim"], rot_dim=case["rot"], value_dim=case["value_dim"], kv_rank=case["rank"],
            scale=(case["head_dim"] + case["rot"]) ** -0.5, window=case["window"], sink=case["sink"],
            exact_weights=case["exact_weights"], position_encoding="rope"),
            name("q", "dkv", "dkv_norm", "uk", "uv", "o", *(["sink"] if case["sink"] else [])))
    if k == "sink":
        return "mixer", PartSpec("sink_window_attention", dict(
            sizes, num_kv_heads=case["kv_heads"], head_dim=case["head_dim"], value_dim=case["value_dim"],
            scale=case["head_dim"] ** -0.5, window=case["window"], keep_first=case["keep_first"], slope_bits=8.0),
            name("q", "k", "v", "o", "g", "q_bias", "k_bias", "v_bias", "temp", "sink"))
    sizes.update(key_dim=case["head_dim"], value_dim=case["value_dim"])
    if k == "gla":
        return "mixer", PartSpec("decay_linear_attention", dict(sizes, decay=None, tau=16.0, decay_rank=16, scale_on="k"),
                                 name("q", "k", "v", "g", "o", "a1", "a2", "a2_bias"))
    if k == "hgrn":
        return "mixer", PartSpec("forget_gate_linear_attention", sizes, name("q", "f", "v", "o", "f_bias", "lower", "norm"))
    return "mixer", PartSpec("gated_delta_rule", dict(sizes, num_qk_heads=case["qk_heads"], taps=case["taps"]),
                             name("q", "k", "v", "g", "b", "a", "q_conv", "k_conv", "v_conv", "a_log", "dt_bias", "norm", "o"))


# ---------------------------------------------------------------------------------------------------
def _cache(case, needs, dtype, pool):
    """A cache that holds the requests' earlier rows, and a slot per request."""
    reqs = _requests(case)
    longest = max(c + n for c, n in reqs)
    cache = PagedCache(needs, PAGE, max(1, _first_pages(case)[1]), len(reqs), longest, dtype, DEV)
    slots = []
    for c, n in reqs:
        slots.append(cache.admit())
        cache.ensure(slots[-1], c + n)
    for g in cache.groups:
        g.pool.copy_(pool)
    return cache, slots


def prepare(case, seed):
    w, rows, pool, residual = _inputs(case, seed)
    dtype = DTYPES[case.get("dtype", "bf16")]
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    if case["kind"] in ("step", "block"):
        arch, cfg = aie.load_config(dict(
            architectures=["LlamaForCausalLM"], hidden_size=case["hidden"], intermediate_size=case["inter"],
            num_hidden_layers=case.get("layers", 1), num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"],
            head_dim=case["head_dim"], vocab_size=case.get("vocab", 64), max_position_embeddings=8192,
            rope_theta=case["theta"], rms_norm_eps=EPS, tie_word_embeddings=False))
        model = Model(arch.build_spec(cfg), dtype, DEV)
        model.load(from_tensors(w, model.tensor_specs(), dtype, model.device))
        cache, slots = _cache(case, model.cache_requests(), dtype, pool)
        steps = [[StepEntry(slots[i], c, rows[i].tolist() if case["kind"] == "step" else [0] * n, [n - 1]) for i, c, n in step]
                 for step in _portions(case)]
        if case["kind"] == "step":
            return dict(kind="step", runner=StepRunner(model, cache), entries=steps[0])
        ctx = StepContext(steps[0], cache, model.device, err, planners=tuple(model.step_planners()))
        return dict(kind="block", model=model, ctx=ctx, caches=cache.layer_cache(0, ctx), stream=torch.cat(rows),
                    pages=cache.groups[0].pool)
    env = BuildEnv(case["hidden"], dtype, torch.device(DEV))
    if case["kind"] == "latent":
        rope = lookup("position_encoding", "rotary")(PartSpec("rotary", dict(rot_dim=case["rot"], theta=500000.0)), env)
        rope.load(None)
        env.position_encodings["rope"] = rope
    family, spec = _spec(case)
    part = lookup(family, spec.kind)(spec, env)
    part.load(from_tensors(w, part.tensor_specs(), dtype, env.device))
    if case["kind"] == "moe":
        return dict(kind="moe", part=part, h=rows[0], ctx=type("Step", (), {"err": err})())
    cache, slots = _cache(case, [CacheNeed(0, "p", part.cache_request(), part.state_request())], dtype, pool)
    planner = part.step_planner()
    steps, at = [], [0] * len(rows)
    for step in _portions(case):
        entries = [StepEntry(slots[i], c, [0] * n, []) for i, c, n in step]
        ctx = StepContext(entries, cache, env.device, err, planners=(planner,) if planner is not None else ())
        h = torch.cat([rows[i][at[i]:at[i] + n] for i, c, n in step])
        for i, c, n in step:
            at[i] += n
        steps.append((h, ctx, cache.layer_cache(0, ctx)["p"]))
    state = cache.state.get((0, "p"))
    out = dict(kind="mixer", part=part, steps=steps, cache=cache, slots=slots if state is not None else [],
               state=state, pages=cache.groups[0].pool if cache.groups else None)
    if all(n == 1 for _, n in _requests(case)):
        # a small step leaves the parts of a split product to the norm that follows it
        norm = lookup("norm", "rmsnorm")(PartSpec("rmsnorm", dict(size=case["hidden"], eps=EPS), dict(weight="w")), env)
        norm.load(from_tensors({"w": torch.ones(case["hidden"], dtype=torch.bfloat16, device=DEV)}, norm.tensor_specs(),
                               dtype, env.device))
        out.update(kind="joined", norm=norm, residual=residual)
    return out


def run(state):
    kind = state["kind"]
    if kind == "step":
        return state["runner"].step(state["entries"])
    if kind == "moe":
        return state["part"].forward(state["h"], state["ctx"])
    if kind == "block":
        model = state["model"]
        x, pending = model.layers[0].block.forward(state["stream"].clone(), None, state["ctx"], state["caches"])
        normed = model.final_norm.forward(x, pending)
        return dict(normed=normed, stream=x, pages=state["pages"])
    for slot in state["slots"]:           # as the engine does for a request it admits
        state["cache"].reset_state(slot)
    outs = [state["part"].forward(h, ctx, lc) for h, ctx, lc in state["steps"]]
    if kind == "joined":
        outs = [state["norm"].forward(state["residual"], outs[0], write_back=False)]
    return dict(out=outs, state=state["state"], pages=state["pages"])


# ---------------------------------------------------------------------------------------------------
def _visible(case, q, k):
    """Mask [len(q), len(k)] of the keys at positions k that queries at positions q read."""
    window, first = case.get("window", 0), case.get("keep_first", 0)
    ok = k[None, :] <= q[:, None]
    if window:
        ok &= (q[:, None] - k[None, :] < window) | (k[None, :] < first)
    return ok


def _pairs(case):
    """Visible (query, key) pairs of all requests."""
    window, first, total = case.get("window", 0), case.get("keep_first", 0), 0
    for c, n in _requests(case):
        for p in range(c, c + n):
            total += min(p + 1, window + min(first, max(0, p + 1 - window))) if window else p + 1
    return total


def work(case):
    k, D = case["kind"], case["hidden"]
    reqs = _requests(case)
    T, cached = sum(n for _, n in reqs), sum(c for c, _ in reqs)
    if k in ("step", "block"):
        H, K, d, F = case["heads"], case["kv_heads"], case["head_dim"], case["inter"]
        es, L, V = (4 if case["dtype"] == "fp32" else 2), case.get("layers", 1), case.get("vocab", 0)
        per = D * d * (2 * H + 2 * K) + 3 * D * F
        logits = len(reqs) if k == "step" else 0
        rows = (T * D * es + logits * V * 4) if k == "step" else T * D * (8 + es)
        return dict(bytes=es * (L * per + V * D * bool(logits)) + L * 2 * K * d * es * (cached + T) + rows,
                    flops=2.0 * T * L * per + 2.0 * logits * V * D + 4.0 * L * _pairs(case) * H * d)
    if k == "moe":
        E, F, Fs = case["experts"], case["inter"], case["shared"]
        return dict(bytes=2 * (3 * D * (E * F + Fs) + E * D) + T * D * 6, flops=2.0 * T * D * (3 * (case["top"] * F + Fs) + E))
    H, e = case["heads"], case["value_dim"]
    if k == "ssm":
        inner, GN = H * e, case["groups"] * case["state"]
        wts = D * (3 * inner + 2 * GN + H)
        return dict(bytes=2 * wts + T * D * 6 + len(reqs) * H * case["state"] * e * 4,
                    flops=2.0 * T * wts + 4.0 * T * H * case["state"] * e)
    d = case["head_dim"]
    if k == "latent":
        rank, rot = case["rank"], case["rot"]
        wts = D * (H * (d + rot) + rank + rot + H * e) + H * rank * (d + e)
        seen = sum(n + (min(c, case["window"] - 1) if case["window"] else c) for c, n in reqs)
        return dict(bytes=2 * wts + T * D * 6 + 2 * (rank + rot) * seen, flops=2.0 * T * wts + 2.0 * _pairs(case) * H * (2 * rank + rot))
    if k == "sink":
        G = case["kv_heads"]
        wts = D * (H * d + G * (d + e) + H + H * e)
        seen = sum(n + min(c, case["window"] + case["keep_first"]) for c, n in reqs)
        return dict(bytes=2 * wts + T * D * 6 + 2 * G * (d + e) * seen, flops=2.0 * T * wts + 2.0 * _pairs(case) * H * (d + e))
    state = len(reqs) * H * d * e * 4
    if k == "delta":
        wts = D * (2 * case["qk_heads"] * d + 3 * H * e + 2 * H)
        return dict(bytes=2 * wts + T * D * 6 + state, flops=2.0 * T * wts + 6.0 * T * H * d * e)
    wts = D * (2 * H * d + (3 if k == "gla" else 2) * H * e) + (16 * (D + H * d) if k == "gla" else 0)
    return dict(bytes=2 * wts + T * D * 6 + state, flops=2.0 * T * wts + 4.0 * T * H * d * e)


# About four times the error of a pass against exact() (2-norms; bfloat16 outputs and, where a layer has them, bfloat16
# products): 0.0044 / 0.0038 / 0.0029 for a chain of layers, the compressed cache and the sink, 0.0026 for a block, the
# state-space layer and the experts, 0.0017 for the other mixers; 2.3e-6 in 32 bits.
_REL = dict(step=1.6e-2, latent=1.5e-2, sink=1.2e-2, block=1e-2, ssm=1e-2, moe=1e-2, gla=7e-3, hgrn=7e-3, delta=7e-3)


def tolerance(case):
    return {"rel": 1e-5 if case.get("dtype") == "fp32" else _REL[case["kind"]]}


# ---------------------------------------------------------------------------------------------------
# the same in 64 bits, plain torch
def _rms(x, w=None):
    y = x * torch.rsqrt((x * x).mean(dim=-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _rope(x, pos, theta):
    """x [tokens, heads, d], split halves; frequencies and angles as float32 numbers, as the architectures define them."""
    half = x.shape[-1] // 2
    i = torch.arange(half, device=x.device, dtype=torch.float32)
    freq = 1.0 / torch.pow(torch.tensor(theta, dtype=torch.float32, device=x.device), 2.0 * i / (2 * half))
    a = (pos.float()[:, None] * freq[None, :]).double()[:, None, :]
    x1, x2 = x[..., :half], x[..., half:]
    return torch.cat([x1 * a.cos() - x2 * a.sin(), x1 * a.sin() + x2 * a.cos()], dim=-1)


def _softmax(s, ok, sink=None):
    """Softmax over the last axis of s [..., q, k] where ok, with an optional leak exp(sink)."""
    s = s.masked_fill(~ok, -math.inf)
    m = s.amax(dim=-1, keepdim=True)
    if sink is not None:
        m = torch.maximum(m, sink)
    p = torch.exp(s - m)
    den = p.sum(dim=-1, keepdim=True)
    return p / (den + torch.exp(sink - m) if sink is not None else den)


def _pages_of(case, i):
    """Places (page, slot) of request i's positions."""
    first = _first_pages(case)[0][i]
    c, n = _requests(case)[i]
    pos = torch.arange(c + n, device=DEV)
    return first + pos // PAGE, pos % PAGE


def _llama_layer(case, w, p, x, pool, run, keep):
    """x: residual rows per request; pool [runs, 2, pages, K, page, d]; keep: float64 pool that receives the new rows."""
    H, K, d = case["heads"], case["kv_heads"], case["head_dim"]
    lin = lambda t, n: t @ w(p + n + ".weight").T
    out = []
    for i, (c, n) in enumerate(_requests(case)):
        h = _rms(x[i], w(p + "input_layernorm.weight"))
        pos = torch.arange(c, c + n, device=DEV)
        q = _rope(lin(h, "self_attn.q_proj").view(n, H, d), pos, case["theta"])
        kn = _rope(lin(h, "self_attn.k_proj").view(n, K, d), pos, case["theta"])
        vn = lin(h, "self_attn.v_proj").view(n, K, d)
        page, slot = _pages_of(case, i)
        ks, vs = (torch.cat([pool[run, z, page[:c], :, slot[:c]].double(), new]) for z, new in ((0, kn), (1, vn)))
        if keep is not None:
            keep[run, 0, page[c:], :, slot[c:]], keep[run, 1, page[c:], :, slot[c:]] = kn, vn
        ok = _visible(case, pos, torch.arange(c + n, device=DEV))
        a = torch.empty(n, H, d, dtype=torch.float64, device=DEV)
        for g in range(K):
            heads = slice(g * (H // K), (g + 1) * (H // K))
            s = torch.einsum("qhd,kd->hqk", q[:, heads], ks[:, g]) * d ** -0.5
            a[:, heads] = torch.einsum("hqk,kd->qhd", _softmax(s, ok), vs[:, g])
        y = x[i] + lin(a.reshape(n, H * d), "self_attn.o_proj")
        h = _rms(y, w(p + "post_attention_layernorm.weight"))
        out.append(y + lin(torch.nn.functional.silu(lin(h, "mlp.gate_proj")) * lin(h, "mlp.up_proj"), "mlp.down_proj"))
    return out


def _conv(x, w, bias=None):
    """Causal convolution over time per channel, zeros before the start, silu; x [n, C], w [C, taps]."""
    taps = w.shape[1]
    pad = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    y = sum(pad[j:j + x.shape[0]] * w[:, j] for j in range(taps))
    return torch.nn.functional.silu(y if bias is None else y + bias), pad[x.shape[0]:]


def _linear_attention(q, k, v, a):
    """q, k, a [n, H, d], v [n, H, e]: outputs [n, H, e] and the last state."""
    S = q.new_zeros(q.shape[1], q.shape[2], v.shape[2])
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * a[t][:, :, None] + k[t][:, :, None] * v[t][:, None, :]
        out[t] = torch.einsum("hde,hd->he", S, q[t])
    return out, S


def _mixer(case, w, h, i, pool, keep):
    """(output rows, state) of request i."""
    k, H, n, silu = case["kind"], case["heads"], h.shape[0], torch.nn.functional.silu
    lin = lambda name: h @ w(name).T
    if k == "ssm":
        e, N, G, inner = case["value_dim"], case["state"], case["groups"], H * case["value_dim"]
        z, xbc, dt = lin("in").split([inner, inner + 2 * G * N, H], dim=1)
        y, tail = _conv(xbc, w("conv"), w("conv_bias"))
        x, B, C = y[:, :inner].view(n, H, e), y[:, inner:inner + G * N].view(n, G, N), y[:, inner + G * N:].view(n, G, N)
        B, C = (t.repeat_interleave(H // G, dim=1) for t in (B, C))
        dt = torch.nn.functional.softplus(dt + w("dt_bias"))
        a = torch.exp(-torch.exp(w("a_log")) * dt)
        o, S = _linear_attention(C, B, x * dt[:, :, None], a[:, :, None].expand(n, H, N))
        o = (o + w("skip")[:, None] * x).reshape(n, inner) * silu(z)
        return (_rms(o.view(n, case["norm_groups"], -1)).reshape(n, inner) * w("norm")) @ w("o").T, dict(tail=tail, S=S)
    d, e = case["head_dim"], case["value_dim"]
    if k == "gla":
        a = torch.sigmoid((h @ w("a1").T) @ w("a2").T + w("a2_bias")) ** (1.0 / 16.0)
        o, S = _linear_attention(lin("q").view(n, H, d), lin("k").view(n, H, d) * d ** -0.5, lin("v").view(n, H, e), a.view(n, H, d))
        return (_rms(o).reshape(n, H * e) * silu(lin("g"))) @ w("o").T, S
    if k == "hgrn":
        f = w("lower") + (1.0 - w("lower")) * torch.sigmoid(lin("f") + w("f_bias"))
        o, S = _linear_attention(silu(lin("q")).view(n, H, d), (1.0 - f).view(n, H, d), lin("v").view(n, H, e), f.view(n, H, d))
        return _rms(o, w("norm")).reshape(n, H * e) @ w("o").T, S
    if k == "delta":
        G = case["qk_heads"]
        x = torch.cat([lin("q"), lin("k"), lin("v")], dim=1)
        y, tail = _conv(x, torch.cat([w("q_conv"), w("k_conv"), w("v_conv")]))
        q, kk, v = y[:, :G * d].view(n, G, d), y[:, G * d:2 * G * d].view(n, G, d), y[:, 2 * G * d:].view(n, H, e)
        unit = lambda t: (t * torch.rsqrt((t * t).sum(dim=-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=1)
        q, kk = unit(q) * d ** -0.5, unit(kk)
        beta = torch.sigmoid(lin("b"))
        g = torch.exp(-torch.exp(w("a_log")) * torch.nn.functional.softplus(lin("a") + w("dt_bias")))
        S, o = h.new_zeros(H, d, e), torch.empty(n, H, e, dtype=h.dtype, device=h.device)
        for t in range(n):
            S = S * g[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.einsum("hde,hd->he", S, kk[t]))
            S = S + kk[t][:, :, None] * u[:, None, :]
            o[t] = torch.einsum("hde,hd->he", S, q[t])
        return (_rms(o, w("norm")).reshape(n, H * e) * silu(lin("g"))) @ w("o").T, dict(tail=tail, S=S)
    c = _requests(case)[i][0]
    pos, keys = torch.arange(c, c + n, device=DEV), torch.arange(c + n, device=DEV)
    ok = _visible(case, pos, keys)
    page, slot = _pages_of(case, i)
    a = torch.empty(n, H, e, dtype=torch.float64, device=DEV)
    if k == "latent":
        rank, rot = case["rank"], case["rot"]
        q, kv = lin("q").view(n, H, d + rot), lin("dkv")
        qr = _rope(q[..., d:], pos, 500000.0)
        new = torch.cat([_rms(kv[:, :rank], w("dkv_norm")), _rope(kv[:, None, rank:], pos, 500000.0)[:, 0]], dim=1)
        rows = torch.cat([pool[0, 0, page[:c], 0, slot[:c]].double(), new])
        keep[0, 0, page[c:], 0, slot[c:]] = new
        for hd in range(H):
            qa = q[:, hd, :d] @ w("uk").view(H, d, rank)[hd]
            s = (qa @ rows[:, :rank].T + qr[:, hd] @ rows[:, rank:].T) * (d + rot) ** -0.5
            p = _softmax(s, ok, w("sink")[hd] if case["sink"] else None)
            a[:, hd] = (p @ rows[:, :rank]) @ w("uv").view(H, e, rank)[hd].T
        return a.reshape(n, H * e) @ w("o").T, None
    G = case["kv_heads"]                                                        # sink
    q = (lin("q") + w("q_bias")).view(n, H, d)
    new = torch.cat([(lin("k") + w("k_bias")).view(n, G, d), _rms((lin("v") + w("v_bias")).view(n, G, e))], dim=2)
    rows = torch.cat([pool[0, 0, page[:c], :, slot[:c]].double(), new])
    keep[0, 0, page[c:], :, slot[c:]] = new
    for hd in range(H):
        g = hd // (H // G)
        s = (q[:, hd] @ rows[:, g, :d].T) * (d ** -0.5 * w("temp")[hd])
        s = s - 2.0 ** (-8.0 * (hd + 1) / H) * (pos[:, None] - keys[None, :])
        a[:, hd] = _softmax(s, ok, w("sink")[hd]) @ rows[:, g, d:]
    return (a * torch.sigmoid(lin("g"))[:, :, None]).reshape(n, H * e) @ w("o").T, None


def _experts(case, w, h):
    T, E, G = h.shape[0], case["experts"], case["groups"]
    silu = torch.nn.functional.silu
    ff = lambda x, p: (silu(x @ w(p + ".gate").T) * (x @ w(p + ".up").T)) @ w(p + ".down").T
    s = torch.sigmoid(h @ w("router").T)
    best = s.view(T, G, E // G).topk(2, dim=2).values.sum(dim=2).topk(case["keep"], dim=1).indices
    open_ = torch.zeros(T, G, dtype=torch.bool, device=h.device).scatter_(1, best, True).repeat_interleave(E // G, dim=1)
    ids = s.masked_fill(~open_, -1.0).topk(case["top"], dim=1).indices
    wt = s.gather(1, ids)
    wt = 2.0 * wt / (wt.sum(dim=1, keepdim=True) + 1e-20)
    out = ff(h, "s")
    for e in range(E):
        t, j = (ids == e).nonzero(as_tuple=True)
        if len(t):
            out.index_add_(0, t, ff(h[t], f"e{e}") * wt[t, j][:, None])
    return out


def exact(case, seed):
    tensors, rows, pool, residual = _inputs(case, seed)
    w = lambda name: tensors[name].double()
    k = case["kind"]
    if k == "moe":
        return _experts(case, w, rows[0].double())
    keep = pool.double() if pool is not None and k != "step" else None
    if k in ("step", "block"):
        x = [w("model.embed_tokens.weight")[r] if k == "step" else r.double() for r in rows]
        for run_ in range(case.get("layers", 1)):
            x = _llama_layer(case, w, f"model.layers.{run_}.", x, pool, run_, keep)
        if k == "step":
            return _rms(torch.cat([r[-1:] for r in x]), w("model.norm.weight")) @ w("lm_head.weight").T
        stream = torch.cat(x)
        return dict(normed=_rms(stream, w("model.norm.weight")), stream=stream, pages=keep)
    done = [_mixer(case, w, r.double(), i, pool, keep) for i, r in enumerate(rows)]
    outs, at = [], [0] * len(rows)
    for step in _portions(case):
        outs.append(torch.cat([done[i][0][at[i]:at[i] + n] for i, _, n in step]))
        for i, _, n in step:
            at[i] += n
    state = None
    if done[0][1] is not None:
        state = {n: torch.stack([s[n] for _, s in done]) for n in done[0][1]} if isinstance(done[0][1], dict) \
            else torch.stack([s for _, s in done])
    if all(n == 1 for _, n in _requests(case)):
        outs = [_rms(residual.double() + outs[0])]
    return dict(out=outs, state=state, pages=keep)
