"""The transforms of line lengths without a compiled plan (radix 16/8/4/2 passes,
then radix 9, then 3; quotients by reciprocals): every count of factors 3,
against numpy's transforms in the packed order (Re 0, Re n/2, Re 1, Im 1, ...).

FP64 directly, within 5e-15 relative L2 (2^-53 times a few operations per pass);
the mixed form's through a projection against the FP64 form's, within 1e-5 (four
FP32 transforms and sweeps, 2^-24 times the tens of operations of each value).
"""
import numpy as np
import pytest

from tests.helpers import case_kwargs, channel_params, rel_l2

pytestmark = pytest.mark.gpu

LENGTHS = [(6, 12), (18, 36), (54, 8), (24, 72), (162, 18), (108, 54), (144, 216), (486, 6), (36, 486),
           (648, 24), (288, 162), (16, 324), (432, 4)]


def packed(x, axis):
    f = np.moveaxis(np.fft.rfft(x, axis=axis), axis, -1)
    n = x.shape[axis]
    out = np.empty(f.shape[:-1] + (n,))
    out[..., 0], out[..., 1] = f[..., 0].real, f[..., n // 2].real
    out[..., 2::2], out[..., 3::2] = f[..., 1:n // 2].real, f[..., 1:n // 2].imag
    return np.moveaxis(out, -1, axis)


@pytest.mark.parametrize("nx,ny", LENGTHS)
def test_fp64_transforms(nx, ny):
    from powerllel_channel_sycl_b200 import Channel
    nz = 6
    with Channel(channel_params(**case_kwargs(nx, ny, nz))) as ch:
        rng = np.random.default_rng(nx * ny)
        p = rng.standard_normal(ch.shape)
        ch.upload("p", p)
        ch.execute_fft_fwd_xpen()
        x = packed(p[1:-1, 1:-1, 1:-1], 2)
        assert rel_l2(ch.download("spec"), x) < 5e-15
        ch.execute_fft_fwd_ypen()
        assert rel_l2(ch.download("spec"), packed(x, 1)) < 5e-15
        ch.execute_fft_bwd_ypen()
        ch.execute_fft_bwd_xpen()
        assert rel_l2(ch.download("p")[1:-1, 1:-1, 1:-1], p[1:-1, 1:-1, 1:-1]) < 1e-14


@pytest.mark.parametrize("nx,ny", [s for s in LENGTHS if s[0] % 4 == 0 and s[1] % 4 == 0])
def test_mixed_projection(nx, ny):
    from powerllel_channel_sycl_b200 import Channel
    rng = np.random.default_rng(nx + ny)
    fields = [rng.uniform(-1, 1, (10, ny + 2, nx + 2)).astype(np.float32) for _ in range(3)]
    got = []
    for precision in (0, 1):
        prm = channel_params(**case_kwargs(nx, ny, 8))
        prm.precision = precision
        with Channel(prm) as ch:
            for name, a in zip("uvw", fields):
                ch.upload(name, a)
            ch.project()
            got.append(np.stack([ch.download(name)[1:-1, 1:-1, 1:-1] for name in "uvw"]))
    assert rel_l2(got[1], got[0]) < 1e-5
