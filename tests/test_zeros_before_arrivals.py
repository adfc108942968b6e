"""Rows that a warp fills with zeros for other warps: one lane arrives on the barrier for all 32, so a __syncwarp() has to stand between the
lanes' stores and that arrival (a vote orders no memory between lanes).  On a GPU the missing order does not show reliably, so the sources
are read."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ai-engine_b200", "csrc")
ZEROS = re.compile(r"make_uint4\(0u?, 0u?, 0u?, 0u?\);")
FENCE = 'asm volatile("fence.proxy.async'
ARRIVES = re.compile(r"\bmbar_(expect_tx|arrive_plain)\(")


def published(text):
    """Per store of zeros that is fenced for copies (shared memory): the text up to the arrival that publishes it."""
    for m in ZEROS.finditer(text):
        arrival = ARRIVES.search(text, m.end())
        if arrival and FENCE in text[m.end():arrival.start()]:
            yield text[m.end():arrival.start()]


@pytest.mark.parametrize("name,places", [("latent_attention_tc.cu", 1), ("attention_prefill_tc.cu", 3)])
def test_zeros_are_ordered_before_the_arrival_of_one_lane(name, places):
    with open(os.path.join(CSRC, name)) as f:
        found = list(published(f.read()))
    assert len(found) == places
    assert all("__syncwarp();" in text for text in found)
