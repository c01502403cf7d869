"""The Thomas sweep with its columns split over the threads of a block
(PLC_TRID=split, and the default where it pays) against the streaming sweep.

Both solve the same systems with the same pivots in different orders of
operations, so both are held to a solution in extended precision (FP64 form) or
in FP64 (mixed form): the split sweep may be a twentieth further off than the
streaming one, plus one rounding of the result.  The sizes are the edges of the
compiled segment lengths (4, 8 and 16 planes for 16 segments, the streaming
sweep above 256 planes), segments left empty or short, lanes that do not fill a
block, fewer than 16 low modes, and a grid whose lanes hold the systems of a
pair in both directions.
"""
import numpy as np
import pytest

from tests.helpers import case_kwargs, channel_params, rel_l2

pytestmark = pytest.mark.gpu

SIZES = [(32, 24, 2), (36, 6, 6), (12, 8, 32), (24, 18, 34), (64, 48, 64), (54, 16, 66), (32, 24, 128),
         (108, 4, 130), (24, 24, 192), (32, 12, 194), (36, 36, 256), (32, 6, 258), (512, 288, 10)]


def channel(monkeypatch, mode, nx, ny, nz, precision=0):
    from powerllel_channel_sycl_b200 import Channel
    monkeypatch.setenv("PLC_TRID", mode)
    prm = channel_params(**case_kwargs(nx, ny, nz))
    prm.precision = precision
    return Channel(prm)


def extended_solution(ch, var):
    """The systems solved in extended precision with exact coefficients."""
    nz, ny, nx = var.shape
    L = np.longdouble
    h = ch.mesh("dzf_global").astype(L)
    lam = []
    for n, size in ((nx, ch.params.lx), (ny, ch.params.ly)):
        m = np.arange(n) // 2
        m[1] = n // 2
        lam.append(2 * (np.cos(2 * np.pi * L(1) * m / n) - 1) * (n / L(size)) ** 2)
    lam = lam[1][:, None] + lam[0][None, :]
    a = [2 / (h[k + 1] * (h[k] + h[k + 1])) for k in range(nz)]
    c = [2 / (h[k + 1] * (h[k + 2] + h[k + 1])) for k in range(nz)]
    a[0] = c[-1] = L(0)
    x = var.astype(L).copy()
    piv = np.empty_like(x)
    b = lam - c[0]
    for k in range(nz):
        if k:
            b = lam - a[k] - c[k] - a[k] * c[k - 1] / piv[k - 1]
            x[k] -= a[k] / piv[k - 1] * x[k - 1]
        piv[k] = b
    piv[nz - 1, 0, 0] = 1  # the singular system is left out of the comparison
    x[nz - 1] /= piv[nz - 1]
    for k in range(nz - 2, -1, -1):
        x[k] = (x[k] - c[k] * x[k + 1]) / piv[k]
    return x


@pytest.mark.parametrize("nx,ny,nz", SIZES)
def test_split_sweep_fp64(monkeypatch, nx, ny, nz):
    var = np.random.default_rng(nz).standard_normal((nz, ny, nx))
    got = {}
    for mode in ("split", "stream"):
        ch = channel(monkeypatch, mode, nx, ny, nz)
        ch.upload("spec", var)
        ch.solve_trid()
        got[mode] = ch.download("spec")
        ref = extended_solution(ch, var)
        ch.close()
    mask = np.ones((ny, nx), bool)
    mask[0, 0] = False
    err = {m: rel_l2(g[:, mask], ref[:, mask]) for m, g in got.items()}
    assert err["split"] <= 1.05 * err["stream"] + 2.0 ** -53, err
    # the singular system of a random right-hand side: the same constant
    assert rel_l2(got["split"][:, 0, 0], got["stream"][:, 0, 0]) < 1e-9


@pytest.mark.parametrize("mode", [None, "split", "tile", "stream"])
@pytest.mark.parametrize("nx,ny,nz", [(32, 24, 2), (64, 48, 64), (36, 6, 10), (32, 6, 258)])
def test_unaligned_array_is_streamed(monkeypatch, nx, ny, nz, mode):
    """An array one element off a 16-byte boundary, whatever the context's sweep: the
    streaming sweep's solution bit for bit."""
    from powerllel_channel_sycl_b200 import Channel
    var = np.random.default_rng(nx).standard_normal((nz, ny, nx))
    ch = channel(monkeypatch, "stream", nx, ny, nz)
    ch.upload("spec", var)
    ch.solve_trid()
    ref = ch.download("spec")
    ch.close()
    monkeypatch.setenv("PLC_TRID", mode) if mode else monkeypatch.delenv("PLC_TRID")
    with Channel(channel_params(**case_kwargs(nx, ny, nz))) as ch:
        field = np.zeros(ch.shape)
        field.ravel()[1:1 + var.size] = var.ravel()
        ch.upload("u1", field)
        ch.solve_trid(ch.ptr("u1") + 8)
        got = ch.download("u1").ravel()
    np.testing.assert_array_equal(got[1:1 + var.size].reshape(var.shape), ref)
    assert got[0] == 0.0 and not got[1 + var.size:].any()


@pytest.mark.parametrize("nx,ny,nz", [s for s in SIZES if s[0] % 4 == 0 and s[1] % 4 == 0])
def test_split_sweep_mixed(monkeypatch, nx, ny, nz):
    monkeypatch.setenv("PLC_FFT_PLANS_F32", "0,0")
    rng = np.random.default_rng(nz + 1)
    fields = [rng.uniform(-1, 1, (nz + 2, ny + 2, nx + 2)) for _ in range(3)]
    fields = [f.astype(np.float32).astype(np.float64) for f in fields]
    got = {}
    for key, mode, precision in (("exact", "stream", 0), ("split", "split", 1), ("stream", "stream", 1)):
        ch = channel(monkeypatch, mode, nx, ny, nz, precision)
        for name, a in zip("uvw", fields):
            ch.upload(name, a)
        ch.project()
        got[key] = np.stack([ch.download(name)[1:-1, 1:-1, 1:-1] for name in "uvw"])
        ch.close()
    err = {m: rel_l2(got[m], got["exact"]) for m in ("split", "stream")}
    assert err["split"] <= 1.05 * err["stream"] + 2.0 ** -24, err


# members whose segments have each compiled length; a column above 256 planes on
# chip or streamed as tuned, and one that only the streaming sweep takes, beside
# short ones; a grid whose own solves take a lane per pair in both directions,
# and one with too few planes for the split sweep to pay
ENSEMBLES = [[(32, 24, 16), (36, 24, 54), (32, 32, 130), (24, 24, 250)],
             [(32, 24, 16), (32, 32, 258), (36, 24, 54), (24, 24, 300)],
             [(512, 288, 64), (32, 24, 16), (512, 288, 10), (24, 24, 258)]]


@pytest.mark.parametrize("chains", [1, 2])
@pytest.mark.parametrize("sizes", ENSEMBLES)
def test_split_sweep_ensemble_matches_alone(monkeypatch, sizes, chains):
    """A member of a batched ensemble takes its own sweep and segment length,
    whatever the other members' columns: the results are those of its own steps."""
    from powerllel_channel_sycl_b200 import Channel, Ensemble
    monkeypatch.setenv("PLC_FFT_PLANS_F32", "0,0")
    monkeypatch.setenv("PLC_RK_KCHUNK_F32", "8")
    prms = []
    for nx, ny, nz in sizes:
        p = channel_params(**case_kwargs(nx, ny, nz))
        p.precision = 1
        prms.append(p)
    alone = []
    for p in prms:
        ch = Channel(p)
        ch.initFlow()
        ch.step(3)
        alone.append([ch.download(f) for f in "uvwp"])
        ch.close()
    ens = Ensemble(prms)
    ens.initFlow()
    ens.set_schedule("batched")
    ens.set_batch_chains(chains)
    ens.step(3)
    for m, ref in zip(ens.members, alone):
        for f, r in zip("uvwp", ref):
            np.testing.assert_array_equal(m.download(f), r)
    ens.close()
