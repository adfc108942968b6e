"""Which form of the 32-bit product a size takes, by the SMs there are: rounds of blocks are counted over the device's own number."""
import ctypes

import pytest

NARROW, AHEAD, WIDE = 0, 1, 2


@pytest.fixture(scope="module")
def form():
    from ai_engine_b200.csrc.build import cuda_library
    return ctypes.CDLL(cuda_library("gemm_f32.cu")).aie_gemm_f32_form


@pytest.mark.parametrize("M,N,batch,sms,want", [
    (64, 9472, 1, 148, AHEAD), (64, 9472, 1, 74, NARROW), (64, 9472, 1, 147, AHEAD),      # 148 blocks (a tenth of a round is let off)
    (64, 9472, 1, 130, NARROW), (64, 4736, 2, 148, AHEAD), (64, 4736, 1, 74, AHEAD),
    (64, 18944, 1, 148, NARROW), (64, 18944, 1, 300, AHEAD), (513, 2048, 1, 148, NARROW), (513, 2048, 1, 300, AHEAD),
    (513, 16384, 1, 148, WIDE), (1, 2048, 1, 148, AHEAD), (1, 2048, 1, 16, NARROW)])
def test_rounds_are_counted_over_the_device_s_sms(form, M, N, batch, sms, want):
    assert form(M, N, batch, sms) == want
