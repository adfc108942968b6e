"""The work lists of latent attention: which portions meet their rows expanded (both forms measured: see the rule), and that the
lists name every token, and every row that an expanded portion reads, exactly once."""
import random
from types import SimpleNamespace

import numpy as np
import pytest

from ai_engine_b200.kernels import ops
from ai_engine_b200.parts.latent_attention import LatentWork


def plan(reqs, H=16, window=0, expands=True):
    cached, lens = (np.array(v, dtype=np.int32) for v in zip(*reqs))
    ctx = SimpleNamespace(h_q_len=lens, h_ctx_len=cached, max_q_len=int(lens.max()), R=len(reqs))
    arrays, scalars = LatentWork(H, window, expands).plan(ctx)
    return SimpleNamespace(**arrays, **scalars)


@pytest.mark.parametrize("H,window,reqs,expanded", [          # us, as they are / expanded
    (16, 0, [(8000, 64)], [False]), (16, 0, [(30000, 96)], [False]), (8, 0, [(3000, 64)], [False]),      # 181 / 260, 718 / 808, 92 / 102
    (16, 0, [(1000, 64)], [True]), (16, 0, [(8000, 128)], [True]), (64, 0, [(8000, 64)], [True]),        # 83 / 71, 301 / 260, 661 / 440
    (16, 0, [(3000, 64)] * 4, [True] * 4), (8, 1024, [(3000, 96)], [True]),                              # 265 / 192, 69 / 61
    (16, 0, [(0, 2048), (30000, 64), (5, 1)], [True, False, False]),                                     # a long tail beside a prompt
    (16, 0, [(0, 63), (9, 1)], [False, False])])
def test_which_portions_are_expanded(H, window, reqs, expanded):
    assert plan(reqs, H, window).expanded.tolist() == expanded
    assert not plan(reqs, H, window, expands=False).expanded.any()


@pytest.mark.parametrize("bound", [1 << 28, 40 << 20, 5 << 20, 1])
def test_lists_name_every_token_and_every_row_once(bound, monkeypatch):
    monkeypatch.setattr(ops, "LATENT_EXPAND_BYTES", bound)
    rng = random.Random(1)
    for _ in range(200):
        window, H = rng.choice([0, 1, 100, 128, 129, 1024]), rng.choice([1, 16, 40])
        reqs = [(rng.randint(0, 2000), rng.choice([1, 1, 3, 64, 65, 300])) for _ in range(rng.randint(1, 40))]
        w = plan(reqs, H, window)
        seen = [(r, off + i) for size, tiles in ((4, w.tiles), (128, w.prompt_tiles)) for r, off in tiles.tolist()
                for i in range(min(size, reqs[r][1] - off))]
        assert sorted(seen) == [(r, i) for r, (_, n) in enumerate(reqs) if n > 1 for i in range(n)]
        assert {r for r, _ in w.prompt_tiles.tolist()} == set(np.flatnonzero(w.expanded).tolist())
        at = 0
        for r in np.flatnonzero(w.expanded).tolist():
            c, n = reqs[r]
            low = max(c - window + 1, 0) // 128 if window else 0
            start = next(g0 for g0, g1, *_ in w.groups if g0 <= at < g1)
            for k in range(low, (c + n - 1) // 128 + 1):
                assert w.gather[at].tolist() == [r, k] and w.row_tile[r] + k == at - start
                at += 1
        ends = [0, 0]
        for g0, g1, p0, p1, heads in w.groups:                    # one behind the other, whole requests, within the bound
            assert [g0, p0] == ends and 1 <= heads <= H and (heads == 1 or (g1 - g0) * heads * 128 * 640 <= bound)
            assert set(w.gather[g0:g1, 0].tolist()) == set(w.prompt_tiles[p0:p1, 0].tolist())
            assert heads == H or len(set(w.gather[g0:g1, 0].tolist())) == 1
            ends = [g1, p1]
        assert ends == [len(w.gather), len(w.prompt_tiles)]
        assert at == len(w.gather) and len(w.row_tile) == (len(reqs) if at else 0)
        assert w.mixed == (bool(at) and not w.expanded.all())
        if w.mixed:                                               # what is not expanded, token behind token
            tokens, t = [], 0
            for r, (_, n) in enumerate(reqs):
                if not w.expanded[r]:
                    assert w.short_start[r] == len(tokens)
                    tokens += range(t, t + n)
                t += n
            assert w.short_tokens.tolist() == tokens and w.n_short == len(tokens)
            assert [w.short_row[i] for i in tokens] == list(range(len(tokens))) and (w.short_row >= 0).sum() == len(tokens)
