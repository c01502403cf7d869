"""The FP64 step's forcing: with x alone forced the bulk mean is taken from the
field that the second RK stage leaves and the correction adds the force; with any
other set of forced components the mean is taken after the correction.

Both against the module entry points called one by one (mean after the
correction): the same operations but for the rounding of the mean, one part in
2^53 of the bulk velocity per step, so three steps agree within 1e-13 relative
L2.  Grids that do not fill the blocks, both block shapes of the RK stages, a
convecting frame.
"""
import numpy as np
import pytest

from tests.helpers import case_kwargs, channel_params, interior, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("forced", [(1, 0, 0), (1, 1, 0), (0, 0, 1), (0, 0, 0)])
@pytest.mark.parametrize("size,u_crf", [((32, 24, 2), 0.0), ((36, 6, 10), 0.3), ((162, 18, 38), 0.0),
                                        ((256, 192, 70), 0.3)])
def test_step_matches_modules(monkeypatch, size, u_crf, forced):
    from powerllel_channel_sycl_b200 import Channel
    monkeypatch.setenv("PLC_FFT_PLANS", "0,0")
    kw = case_kwargs(*size, u_crf=u_crf, is_forced=forced, vel_force=(1.0, 0.01, 0.001))
    a, b = Channel(channel_params(**kw)), Channel(channel_params(**kw))
    rng = np.random.default_rng(size[2])
    for name in "uvw":
        f = rng.uniform(-0.3, 0.3, a.shape) + (name == "u")
        for ch in (a, b):
            ch.upload(name, f)
    for ch in (a, b):
        ch.finish_input()
    a.step(3)
    for _ in range(3):
        b.timeIntVelRK1()
        b.updateBoundVel(None, "u1", "v1", "w1")
        b.timeIntVelRK2()
        b.updateBoundVel()
        b.calcRHS()
        b.execute_poisson_solver()
        b.updateBoundP()
        b.correctVel()
        force = b.forceVel()
        b.updateBoundVel()
    for name in "uvw":
        assert rel_l2(a.download(name), b.download(name)) < 1e-13, name
        assert rel_l2(interior(a.download(name)), interior(b.download(name))) < 1e-13, name
    assert np.abs(a.step_forcing()[1] - force).max() <= 1e-13
    assert a.kernels_per_step == (9 if any(forced) else 8)
    a.close()
    b.close()
