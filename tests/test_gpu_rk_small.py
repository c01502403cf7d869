"""The RK stages of small grids: blocks that march a part of eight planes and
write their halo images inline (chosen at creation) against eight-plane
blocks (pinned), over grids with rows and planes that do not fill a block.

FP64: every point is computed by the same operations whatever block it falls
in, so all fields with their halos are equal.  Mixed: the same but for the bulk
mean, whose per-block sums round in FP32: the velocity agrees within 2e-6
relative L2, the mixed form's bar for the chunk.
"""
import numpy as np
import pytest

from tests.helpers import case_kwargs, channel_params, rel_l2

pytestmark = pytest.mark.gpu

SIZES = [(32, 24, 2), (36, 6, 10), (64, 18, 16), (24, 36, 38), (128, 64, 64)]


def fields(monkeypatch, precision, size, u_crf, pin):
    from powerllel_channel_sycl_b200 import Channel
    for var, val in (("PLC_FFT_PLANS", "0,0"), ("PLC_FFT_PLANS_F32", "0,0"), ("PLC_RK2_CARRY", "0")):
        monkeypatch.setenv(var, val)
    for var in ("PLC_RK_KCHUNK", "PLC_RK_KCHUNK_F32"):
        monkeypatch.setenv(var, "8") if pin else monkeypatch.delenv(var, raising=False)
    prm = channel_params(**case_kwargs(*size, u_crf=u_crf))
    prm.precision = precision
    with Channel(prm) as ch:
        ch.initFlow()
        ch.step(3)
        return [ch.download(f) for f in ("u1", "v1", "w1", "u", "v", "w")]


@pytest.mark.parametrize("u_crf", [0.0, 0.4])
@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("precision", [0, 1])
def test_small_grid_blocks(monkeypatch, precision, size, u_crf):
    if precision and (size[0] % 4 or size[1] % 4):
        pytest.skip("the mixed form needs nx and ny divisible by 4")
    own = fields(monkeypatch, precision, size, u_crf, False)
    ref = fields(monkeypatch, precision, size, u_crf, True)
    for a, b in zip(own, ref):
        if precision:
            assert rel_l2(a, b) <= 2e-6
        else:
            np.testing.assert_array_equal(a, b)
