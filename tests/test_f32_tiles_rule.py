"""When float32 portions beside lone tokens go in tiles: only where two kernels behind one another take less than one."""
import numpy as np
import pytest

from ai_engine_b200.kernels import ops


@pytest.mark.parametrize("reqs,pays", [
    ([(500, 1)] * 16 + [(500, 8)], False),                  # measured: 929 us in two kernels, 847 in one
    ([(0, 384), (100, 129)], True), ([(1000, 8)], True),    # no lone token: 1,056 against 759
    ([(30, 1)] * 4 + [(3000, 300)], True), ([(4000, 1)] * 2 + [(4000, 8)], False), ([(200, 1)] * 64 + [(0, 1500)], True)])
def test_portions_beside_lone_tokens(reqs, pays):
    cached, lens = (np.array(v) for v in zip(*reqs))
    assert ops.f32_tiles_pay(lens, cached, 32, 64, 0) is pays
    assert ops.f32_tiles_pay(lens, cached, 32, 64, 1 << 20) is pays
