"""The generator's convolutions and weight gradients over halo tiles, at every
channel count they are compiled for and at grids whose planes are smaller
than, not a multiple of, and several times a tile.  In the case of 256 cells the halo
tile of the finest level's 128-channel layers does not fit the shared memory
(2 (128 + 2) (256 + 2 (256 + 3)) + 18 * 128 * 16 bytes and more, of 225 KB): those
layers, forward, output and input gradient, take the im2col convolution, as do
the 112-channel layers of the last case, whose tiles would be read in seven parts.

Weights with three terms of +-1 or +-1/2 per output, FiLM tables of eighths and
r = +-1/2: every FP32 sum of the forward pass is exact up to its last bit, so
that a BF16 rounding differs from the oracle's only when it falls within
2^-24 of a tie: on about 2^-15 of the activations of a layer, by 2^-9 each, under
1e-4 over the nine layers.  The gradients add FP32 sums over the voxels and FP32
loss coefficients (2^-22 and the roundings they move): under 1e-3.
"""
import numpy as np
import pytest

from oracle import gen_oracle as go

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


def exact_params(cfg, rng):
    parts = []
    for ci, co, _, act in go.layer_list(cfg):
        w = np.zeros((27, co, ci), np.float32)
        for o in range(co if act else 3):
            for _ in range(3):
                w[rng.integers(27), o, rng.integers(ci)] = rng.choice([-1.0, 1.0, -0.5, 0.5])
        parts.append(w.ravel())
    for _, co, lv, _ in go.layer_list(cfg):
        z = go.level_dims(cfg, lv)[0]
        parts.append(rng.integers(-2, 3, 4 * z * co).astype(np.float32) / 8)
    return np.concatenate(parts)


@pytest.mark.parametrize("nx,ny,nz,channels,latent", [
    (8, 8, 8, [128, 112, 96, 80], 16),     # planes of one voxel at level 0
    (24, 16, 8, [64, 48, 32, 16], 32),     # three voxels in x
    (64, 16, 16, [16, 32, 80, 64], 16),    # five tiles in a plane
    (16, 48, 8, [48, 96, 128, 112], 128),  # long in y
    (128, 8, 8, [112, 16, 16, 48], 48),    # the longest rows that two buffers hold
    (64, 48, 8, [32, 48, 64, 32], 16),     # planes of the default grid
    (256, 8, 8, [16, 16, 32, 128], 16),    # 128 channels of a row too long for the shared memory
    (64, 16, 8, [128, 96, 64, 128], 16),   # one block per SM, 32 of 128 channels each
    (64, 40, 8, [128, 96, 64, 112], 16),   # 112 channels: seven blocks would read each tile
])
def test_halo_tiles_match_oracle(nx, ny, nz, channels, latent):
    from powerllel_channel_sycl_b200.learned import Generator, config
    cfg = dict(nx=nx, ny=ny, nz=nz, channels=channels, latent_channels=latent, batch=2)
    g = Generator(config(**cfg, seed=3))
    rng = np.random.default_rng(nx + ny)
    p = exact_params(cfg, rng)
    g.params = p
    targets = rng.normal(0, 0.02, (2, nz, go.NSTAT))
    targets[..., 0] += np.linspace(0.2, 1.0, nz)
    targets[..., 3:6] += 0.01
    re = np.array([190.0, 330.0])
    g.set_targets(re, targets)
    r = (re - 260) / 140
    out, saved = go.forward(cfg, p.astype(np.float64), g.latent(7), r, bf16=True)
    assert rel(g.forward(re, seed=7), out[..., :3]) < 1e-4
    loss, grad = g.loss_grad(np.array([0, 1], np.int32), re, seed=7)
    sc_mean = np.sqrt(np.mean(targets[..., 0] ** 2))
    sc_var = np.sqrt(np.mean(targets[..., 3] ** 2))
    lref, dout = go.loss_and_dout(out, targets, sc_mean, sc_var)
    gref = go.backward(cfg, p.astype(np.float64), saved, r, dout, bf16=True)
    assert abs(loss - lref) <= 1e-3 * lref
    off = 0
    for ci, co, lv, act in go.layer_list(cfg):
        n = 27 * ci * co
        if np.linalg.norm(gref[off:off + n]) > 0:
            assert rel(grad[off:off + n], gref[off:off + n]) < 1e-3, (ci, co, lv)
        off += n
    assert rel(grad, gref) < 1e-3


@pytest.mark.parametrize("nx,ny,nz", [(8, 8, 8), (64, 16, 16), (24, 24, 8)])
def test_more_latent_channels_forward_only(nx, ny, nz):
    """Above 128 latent channels the forward pass runs and gradients are refused,
    whether the coarsest grid admits halo tiles or not."""
    from powerllel_channel_sycl_b200 import PlcError
    from powerllel_channel_sycl_b200.learned import Generator, config
    g = Generator(config(nx=nx, ny=ny, nz=nz, channels=[16, 16, 16, 16], latent_channels=144, batch=1,
                         seed=3))
    g.set_targets([180.0], np.full((1, nz, go.NSTAT), 0.1))
    assert np.isfinite(g.forward([180.0], seed=7)).all()
    with pytest.raises(PlcError, match="weight gradient"):
        g.loss_grad(np.array([0], np.int32), [180.0], seed=7)
    with pytest.raises(PlcError, match="weight gradient"):
        g.train(1)
