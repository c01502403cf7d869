"""The RK stages of small grids: blocks that march 2 or 4 planes, and halo
images written inline by whole warps, over grids with rows and planes that do
not fill a block.  Every chunk is pinned in turn.

FP64: the first stage and the boundary update, run one by one through the module
entry points (a kernel that writes no halo, and the boundary kernel), give
every value of u1, v1, w1 with its halo: equal, the operations being the same.
The second stage's halo is overwritten within the step, but the divergence next
to the faces is taken from it: the pressure agrees with the module path's within
1e-10 (rounding of 2^-53, amplified up to 1e4 times, twice over), the velocity
within 1e-13.

Mixed: halos equal what the interior values ask for (periodic images, ghosts
2 bc - v of u and v and the wall value of w, one FP32 rounding), and the
interiors agree with the FP64 form after one step within the form's bars, 1e-4
for the velocity and 5e-3 for the pressure up to a constant.
"""
import numpy as np
import pytest

from tests.helpers import case_kwargs, channel_params, demean, interior, rel_l2

pytestmark = pytest.mark.gpu

SIZES = [(32, 24, 2), (36, 6, 10), (64, 18, 16), (24, 36, 38), (128, 64, 64)]


def channel(monkeypatch, precision, size, u_crf, chunk):
    from powerllel_channel_sycl_b200 import Channel
    for var, val in (("PLC_FFT_PLANS", "0,0"), ("PLC_FFT_PLANS_F32", "0,0"), ("PLC_RK2_CARRY", "0")):
        monkeypatch.setenv(var, val)
    for var in ("PLC_RK_KCHUNK", "PLC_RK_KCHUNK_F32"):
        monkeypatch.setenv(var, str(chunk))
    prm = channel_params(**case_kwargs(*size, u_crf=u_crf))
    prm.precision = precision
    ch = Channel(prm)
    assert ch.rk_kchunk == min(chunk, size[2])
    rng = np.random.default_rng(size[2])
    for name in "uvw":
        f = rng.uniform(-0.3, 0.3, ch.shape) + (name == "u")
        ch.upload(name, f.astype(np.float32))  # the same values in both forms
    ch.finish_input()
    return ch


def with_halo(name, a, u_crf):
    """The field that the interior of `a` and the boundary conditions give, in a's type."""
    out = np.zeros_like(a)
    out[1:-1, 1:-1, 1:-1] = a[1:-1, 1:-1, 1:-1]
    x = a.dtype.type
    if name[0] == "w":
        out[0], out[-2], out[-1] = x(0), x(0), x(0)
    else:
        bc = x(-u_crf) if name[0] == "u" else x(0)
        out[0], out[-1] = x(2) * bc - out[1], x(2) * bc - out[-2]
    out[:, 0], out[:, -1] = out[:, -2], out[:, 1]
    out[:, :, 0], out[:, :, -1] = out[:, :, -2], out[:, :, 1]
    return out


@pytest.mark.parametrize("chunk", [2, 4, 8])
@pytest.mark.parametrize("u_crf", [0.0, 0.4])
@pytest.mark.parametrize("size", SIZES)
def test_small_grid_blocks_fp64(monkeypatch, size, u_crf, chunk):
    a = channel(monkeypatch, 0, size, u_crf, chunk)
    b = channel(monkeypatch, 0, size, u_crf, 8)
    a.step(1)
    b.timeIntVelRK1()
    b.updateBoundVel(None, "u1", "v1", "w1")
    b.timeIntVelRK2()
    b.updateBoundVel()
    b.calcRHS()
    b.execute_poisson_solver()
    b.updateBoundP()
    b.correctVel()
    b.forceVel()
    b.updateBoundVel()
    for name in ("u1", "v1", "w1"):
        np.testing.assert_array_equal(a.download(name), b.download(name), name)
    assert rel_l2(demean(a.download("p")), demean(b.download("p"))) < 1e-10
    for name in "uvw":
        got = a.download(name)
        assert rel_l2(got, b.download(name)) < 1e-13, name
        np.testing.assert_array_equal(got, with_halo(name, got, u_crf), name)
    a.close()
    b.close()


@pytest.mark.parametrize("chunk", [2, 4, 8])
@pytest.mark.parametrize("u_crf", [0.0, 0.4])
@pytest.mark.parametrize("size", [s for s in SIZES if s[0] % 4 == 0 and s[1] % 4 == 0])
def test_small_grid_blocks_mixed(monkeypatch, size, u_crf, chunk):
    a = channel(monkeypatch, 1, size, u_crf, chunk)
    b = channel(monkeypatch, 0, size, u_crf, 8)
    for ch in (a, b):
        ch.step(1)
    for name in ("u1", "v1", "w1", "u", "v", "w"):
        got = a.download(name)
        single = got.astype(np.float32)
        np.testing.assert_array_equal(single, with_halo(name, single, u_crf), name)
        assert rel_l2(interior(got), interior(b.download(name))) <= 1e-4, name
    assert rel_l2(demean(a.download("p")), demean(b.download("p"))) <= 5e-3
    a.close()
    b.close()
