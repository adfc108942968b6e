"""How portions are spread over launches whose scratch has a bound: every portion and head once, in order, within the bound."""
import random

import numpy as np

from ai_engine_b200.kernels import ops


def test_every_portion_and_head_once_within_the_bound():
    rng = random.Random(3)
    for _ in range(300):
        lens = np.array([rng.choice([1, 7, 64, 65, 500, 5000]) for _ in range(rng.randint(1, 40))])
        H, head_bytes, budget, least = rng.choice([1, 6, 64, 3000]), rng.randint(1, 50), rng.choice([1, 100, 10000, 10 ** 9]), rng.choice([8, 65])
        seen, chunks_of = [], lambda n: (n + 63) // 64
        for r0, r1, portions, chunks, head0, heads in ops._portion_ranges(lens, least, H, head_bytes, budget):
            mine = [r for r in range(r0, r1) if lens[r] >= least]
            assert mine[0] == r0 and mine[-1] == r1 - 1 and portions == len(mine) and chunks == sum(chunks_of(int(lens[r])) for r in mine)
            assert portions * heads <= 65535 and 1 <= heads and head0 + heads <= H
            assert chunks * heads * head_bytes <= budget or (portions == 1 and heads == 1)
            seen += [(r, h) for r in mine for h in range(head0, head0 + heads)]
        assert sorted(seen) == [(r, h) for r in range(len(lens)) if lens[r] >= least for h in range(H)]
