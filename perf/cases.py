"""The calls that a user's program spends its GPU time in, as measurable cases.

listed() names them, draw() gives further ones of the same ranges, prepare()
builds what a program holds before the call (contexts, fields, weights), run()
is one pass through the package's public entry points, work() the bytes and
operations such a pass cannot do without, exact() what run() returns in plain
64-bit torch.

Kinds of case:

step      Channel.step: the fused time step, both precision forms, from the
          smallest grid that is run (32 x 24 x 16) to the largest
          (768 x 384 x 256); options: a CFL-controlled dt, a convecting frame
          (u_crf), the spin-up judge's samples after the steps (Re_tau and
          the mean profile), running statistics sampled between the steps.
modules   the time loop of a program that calls the module entry points one
          by one, as the reference's main program does.
ensemble  Ensemble.step: independent channels of uneven grids stepped together.
propose   Generator.propose: the learned initialiser's inference, the
          interpolation onto the channel's grid and the solver's projection.
train     Generator.train: iterations of the learned initialiser's training.

The velocities are the state that a run is continued from, and every case
that advances a channel returns them whole.  The pressure follows from them in
every step and is defined only up to the free constant of the singular
(0,0) mode, which is round-off in the FP64 form: its gradient enters the
velocities, and that is where it is compared.
"""
import math

import numpy as np
import torch

from powerllel_channel_sycl_b200 import Channel, Ensemble, learned, make_params

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
TWO_PI = 2.0 * math.pi
FIELDS = ("u", "v", "w")


# ---- the cases ------------------------------------------------------------------
def listed():
    return [
        # a first trial of a set-up, and the size of unit tests: launches and latency only
        {"name": "step_fp64_32x24x16", "kind": "step", "form": "fp64", "nx": 32, "ny": 24, "nz": 16,
         "steps": 20, "cfl": 0.0, "u_crf": 0.0, "judge": False, "stats": False},
        # Re_tau 180 on the grid that the reference runs on a CPU, fixed dt
        {"name": "step_fp64_128x64x64", "kind": "step", "form": "fp64", "nx": 128, "ny": 64, "nz": 64,
         "steps": 20, "cfl": 0.0, "u_crf": 0.0, "judge": False, "stats": False},
        # a grid chosen for a resolution and not for its factors (3^3 * 4, 3^2 * 8, 3^3 * 2)
        {"name": "step_mixed_108x72x54", "kind": "step", "form": "mixed", "nx": 108, "ny": 72, "nz": 54,
         "steps": 20, "cfl": 0.5, "u_crf": 0.0, "judge": False, "stats": False},
        # another, in FP64, with a length of 2 * 3^4
        {"name": "step_fp64_162x108x90", "kind": "step", "form": "fp64", "nx": 162, "ny": 108, "nz": 90,
         "steps": 20, "cfl": 0.5, "u_crf": 0.0, "judge": False, "stats": False},
        # the spin-up loop at Re_tau 180: 20 steps, then the judge's samples
        {"name": "spinup_mixed_256x192x128", "kind": "step", "form": "mixed", "nx": 256, "ny": 192,
         "nz": 128, "steps": 20, "cfl": 0.4, "u_crf": 0.0, "judge": True, "stats": False},
        # a production run at Re_tau 180 in a convecting frame with statistics every 10 steps
        {"name": "stats_fp64_256x192x128", "kind": "step", "form": "fp64", "nx": 256, "ny": 192, "nz": 128,
         "steps": 20, "cfl": 0.5, "u_crf": 0.5, "judge": False, "stats": True},
        # Re_tau 550, the largest grid, in both forms
        {"name": "step_fp64_768x384x256", "kind": "step", "form": "fp64", "nx": 768, "ny": 384, "nz": 256,
         "steps": 10, "cfl": 0.5, "u_crf": 0.0, "judge": False, "stats": False},
        {"name": "step_mixed_768x384x256", "kind": "step", "form": "mixed", "nx": 768, "ny": 384, "nz": 256,
         "steps": 10, "cfl": 0.5, "u_crf": 0.0, "judge": False, "stats": False},
        # a program written against the reference's modules
        {"name": "modules_fp64_192x96x96", "kind": "modules", "nx": 192, "ny": 96, "nz": 96, "steps": 10},
        # a parameter study, and the training data of the learned initialiser
        {"name": "ensemble_mixed_16", "kind": "ensemble", "members": 16, "specs": 3, "steps": 20},
        # the learned initialiser at work, and its training
        {"name": "propose_256x192x128", "kind": "propose", "nx": 256, "ny": 192, "nz": 128, "re_tau": 180.0},
        {"name": "train_64x48x64_b4", "kind": "train", "batch": 4, "iters": 5},
    ]


# line lengths of the repository's configurations and tests, and odd ones between them
NX = (32, 36, 48, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256, 288, 324, 384, 432, 512, 648, 768)
NY = (24, 32, 36, 48, 54, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256, 288, 324, 384)
NZ = (16, 30, 38, 48, 54, 64, 74, 90, 96, 110, 128, 150, 160, 192, 218, 256)


def _draw_grid(rng, least, most, four):
    """A grid whose number of points is spread over the logarithm of the range."""
    want = math.exp(rng.uniform(math.log(least), math.log(most)))
    best = None
    for _ in range(60):
        g = rng.choice(NX), rng.choice(NY), rng.choice(NZ)
        if four and (g[0] % 4 or g[1] % 4):
            continue
        off = abs(math.log(g[0] * g[1] * g[2] / want)) + max(0.0, g[1] / g[0] - 1.5)
        if g[0] * g[1] * g[2] <= most and (best is None or off < best[0]):
            best = off, g
    return best[1]


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["modules", "ensemble", "propose", "train"])
    if kind == "step":
        form = rng.choice(["fp64", "mixed"])
        nx, ny, nz = _draw_grid(rng, 12288, 768 * 384 * 256, form == "mixed")
        points = nx * ny * nz
        return {"kind": "step", "form": form, "nx": nx, "ny": ny, "nz": nz,
                "steps": 20 if points < 2e7 else 10,
                "cfl": rng.choice([0.4, 0.5]), "u_crf": rng.choice([0.0, 0.0, 0.5]),
                "judge": rng.random() < 0.3, "stats": points < 2e7 and rng.random() < 0.3}
    if kind == "modules":
        nx, ny, nz = _draw_grid(rng, 12288, 256 * 192 * 128, False)
        return {"kind": "modules", "nx": nx, "ny": ny, "nz": nz, "steps": 10}
    if kind == "ensemble":
        return {"kind": "ensemble", "members": rng.randint(3, 16), "specs": rng.randint(4, 99), "steps": 20}
    if kind == "propose":
        nx, ny, nz = rng.choice([(128, 96, 64), (192, 144, 128), (256, 192, 128), (216, 108, 64)])
        return {"kind": "propose", "nx": nx, "ny": ny, "nz": nz, "re_tau": round(rng.uniform(120.0, 400.0), 1)}
    return {"kind": "train", "batch": rng.randint(1, 4), "iters": rng.randint(2, 5)}


# ---- parameters of a case ---------------------------------------------------------
def _physics(nx, ny, nz):
    """Re_tau 550's box above 30 million points, Re_tau 180's below."""
    if nx * ny * nz > 30e6:
        return dict(lx=TWO_PI, ly=math.pi, lz=2.0, re=10000.0, stretch_ratio=1.8)
    return dict(lx=2 * TWO_PI, ly=TWO_PI, lz=2.0, re=2800.0, stretch_ratio=1.5)


def _params(nx, ny, nz, form, nt_check, cfl, u_crf=0.0, physics=None, stats=False):
    return make_params(nx=nx, ny=ny, nz=nz, mesh_type=1, stretch_func=0, u_ref=1.0, l_ref=1.0, dt=2e-3,
                       nt_check=nt_check, cfl_limit=1.0, div_limit=1e-6, initial_field="poi",
                       init_with_noise=1, noise_intensity=0.1, is_forced=[1, 0, 0],
                       vel_force=[1.0, 0.0, 0.0], precision=form, cfl_target=cfl, u_crf=u_crf,
                       sample_interval=10, stat_which_var=[1] * 9 + [0, 0] if stats else [0] * 11,
                       **(physics or _physics(nx, ny, nz)))


def _member_specs(seed, n):
    """Uneven channels between 64 x 48 x 48 and 256 x 192 x 128, Re_tau in [120, 400]."""
    rng = np.random.default_rng(seed)
    out = []
    while len(out) < n:
        nx, ny, nz = (int(rng.choice(c)) for c in ((64, 96, 128, 192, 256), (48, 64, 96, 128, 192),
                                                   (48, 64, 96, 128)))
        if nx < ny / 2:
            continue
        re = learned.re_from_re_tau(float(rng.uniform(120.0, 400.0)))
        out.append((nx, ny, nz, dict(lx=2 * TWO_PI, ly=TWO_PI, lz=2.0, re=re, stretch_ratio=1.5)))
    return out


# ---- inputs -----------------------------------------------------------------------
def _mesh(nz, lz, ratio):
    """Cell heights with one ghost cell per wall, and the centres (tanh stretching)."""
    z = torch.arange(nz + 1, dtype=torch.float64, device=DEVICE) / nz
    zf = 0.5 * (1.0 + torch.tanh((z - 0.5) * ratio) / math.tanh(ratio / 2.0))
    h = lz * (zf[1:] - zf[:-1])
    h = torch.cat([h[:1], h, h[-1:]])
    return h, lz * 0.5 * (zf[1:] + zf[:-1])


def _start_fields(nx, ny, nz, phys, form, seed):
    """The laminar profile of bulk velocity 1 and seeded cell noise of amplitude 0.1, (nz, ny, nx)."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    _, zc = _mesh(nz, phys["lz"], phys["stretch_ratio"])
    z = (zc / phys["lz"])[:, None, None]
    out = []
    for q in range(3):
        a = torch.rand((nz, ny, nx), generator=g, dtype=torch.float64, device=DEVICE)
        a.mul_(0.2).sub_(0.1)
        if q == 0:
            a += 6.0 * z * (1.0 - z)
        out.append(a.float() if form == "mixed" else a)
    return out


class _Memory:
    """Device memory of a context for torch.as_tensor, without a copy."""

    def __init__(self, ptr, shape, kind, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": kind, "data": (ptr, False), "version": 3}


def _interior(ch, field):
    """A view of a field's interior, (nz, ny, nx)."""
    if ch.mixed:
        ptr, _, pitch = ch.ptr_f32(field)
        a = torch.as_tensor(_Memory(ptr, (ch.nz + 2, ch.ny + 2, pitch), "<f4", ch), device=DEVICE)
    else:
        a = torch.as_tensor(_Memory(ch.ptr(field), ch.shape, "<f8", ch), device=DEVICE)
    return a[1:-1, 1:-1, 1:ch.nx + 1]


def _fill(ch, phys, form, seed):
    for name, a in zip(FIELDS, _start_fields(ch.nx, ch.ny, ch.nz, phys, form, seed)):
        _interior(ch, name).copy_(a)
    torch.cuda.synchronize()
    ch.finish_input()


def _start_params(seed):
    """The generator's parameters before training: He-normal weights (none for the output's
    unused channels) and no conditioning, as one flat FP32 vector."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    layers, parts = _gen_layers(), []
    for ci, co, _ in layers:
        sd = math.sqrt((1.0 if co == 16 else 2.0) / (27 * ci))
        w = sd * torch.randn((27, co, ci), generator=g, dtype=torch.float32, device=DEVICE)
        if co == 16:
            w[:, 3:] = 0.0
        parts.append(w.flatten())
    parts += [torch.zeros(4 * (64 >> (3 - lv)) * co, device=DEVICE) for _, co, lv in layers]
    return torch.cat(parts)


def _grid(case):
    return case["nx"], case["ny"], case["nz"]


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "seed": int(seed)}
    if kind in ("step", "modules"):
        form = case.get("form", "fp64")
        phys = _physics(*_grid(case))
        ch = Channel(_params(*_grid(case), form, case["steps"], case.get("cfl", 0.0), case.get("u_crf", 0.0),
                             stats=case.get("stats", False)))
        _fill(ch, phys, form, seed)
        if case.get("stats"):
            ch.initStat()
        state["fields"] = [_interior(ch, f) for f in FIELDS]
        state["ch"], state["nt"] = ch, 0
        state["kind"] = np.float32 if ch.mixed else np.float64  # what its fields hold
    elif kind == "ensemble":
        specs = _member_specs(case["specs"], case["members"])
        ens = Ensemble([_params(nx, ny, nz, "mixed", case["steps"], 0.5, physics=phys)
                        for nx, ny, nz, phys in specs])
        ens.autotune(steps=3)
        for i, (m, spec) in enumerate(zip(ens.members, specs)):
            _fill(m, spec[3], "mixed", 1000 * int(seed) + i)
        state["fields"] = [[_interior(m, f) for f in FIELDS] for m in ens.members]
        state["ens"] = ens
    elif kind == "propose":
        ch = Channel(_params(*_grid(case), "mixed", 100, 0.4))
        state["fields"] = [_interior(ch, f) for f in FIELDS]
        state["ch"], state["gen"] = ch, learned.load_weights()
    elif kind == "train":
        gen = learned.Generator(learned.config(batch=case["batch"]))
        gen.params = _start_params(seed).cpu().numpy()
        d = np.load(learned.TARGETS)
        gen.set_targets(d["re_tau"], d["stats"])
        state["gen"] = gen
    return state


# ---- one pass -----------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        ch = state["ch"]
        out = dict(zip(FIELDS, state["fields"]))
        if case["stats"]:
            for _ in range(case["steps"] // 10):
                ch.step(10)
                state["nt"] += 10
                ch.calcStat(state["nt"])
            mean = ch.stat_profiles()
            out["stats"] = np.stack([mean[name] for name in ch.STAT_NAMES[:9]]).astype(state["kind"])
        else:
            ch.step(case["steps"])
        if case["judge"]:
            out["judged"] = np.append(ch.mean_profile(), ch.re_tau() / 180.0).astype(state["kind"])
        return out
    if kind == "modules":
        ch = state["ch"]
        for _ in range(case["steps"]):
            ch.timeIntVelRK1()
            ch.updateBoundVel(u="u1", v="v1", w="w1")
            ch.timeIntVelRK2()
            ch.updateBoundVel()
            ch.calcRHS()
            ch.execute_poisson_solver()
            ch.updateBoundP()
            ch.correctVel()
            ch.forceVel()
            ch.updateBoundVel()
        ch.sync()
        return dict(zip(FIELDS, state["fields"]))
    if kind == "ensemble":
        state["ens"].step(case["steps"])
        return state["fields"]
    if kind == "propose":
        state["gen"].propose(state["ch"], case["re_tau"], seed=state["seed"] & 0xFFFF)
        return dict(zip(FIELDS, state["fields"]))
    loss = state["gen"].train(case["iters"], lr=1e-3, seed=state["seed"] & 0xFFFF)
    # the network computes its outputs in 32 bits and less
    return {"loss": loss.astype(np.float32), "params": state["gen"].params}


# ---- bytes and operations that a pass cannot do without ------------------------------
def _step_work(nx, ny, nz, size):
    """One time step: u, v, w read, u, v, w, p written; the two stages' stencils, the
    four real transforms and the sweep."""
    n = nx * ny * nz
    return 7.0 * size * n, n * (2 * 180.0 + 2 * 2.5 * (math.log2(nx) + math.log2(ny)) + 8.0 + 20.0)


def _gen_layers(cfg_channels=(128, 96, 64, 32), latent=16):
    """(ci, co, level) of the generator's convolutions; level 3 is the 64 x 48 x 64 grid."""
    out = [(latent, cfg_channels[0], 0), (cfg_channels[0], cfg_channels[0], 0)]
    for lv in range(1, 4):
        out += [(cfg_channels[lv - 1], cfg_channels[lv], lv), (cfg_channels[lv], cfg_channels[lv], lv)]
    return out + [(cfg_channels[3], 16, 3)]


def _gen_work(batch):
    """Operations of a forward pass; bytes of its weights, activations and output."""
    flops, size = 0.0, 0.0
    for ci, co, lv in _gen_layers():
        voxels = batch * (64 * 48 * 64) / 8 ** (3 - lv)
        flops += 2.0 * 27 * ci * (co if co != 16 else 3) * voxels
        size += 27 * ci * co * 2.0
    return flops, size + batch * 64 * 48 * 64 * 3 * 4.0


def work(case):
    kind = case["kind"]
    if kind in ("step", "modules"):
        b, f = _step_work(*_grid(case), 4 if case.get("form") == "mixed" else 8)
        return {"bytes": b * case["steps"], "flops": f * case["steps"]}
    if kind == "ensemble":
        parts = [_step_work(nx, ny, nz, 4) for nx, ny, nz, _ in _member_specs(case["specs"], case["members"])]
        return {"bytes": case["steps"] * sum(p[0] for p in parts), "flops": case["steps"] * sum(p[1] for p in parts)}
    if kind == "propose":
        flops, size = _gen_work(1)
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": size + 4.0 * 4 * n, "flops": flops + n * (40.0 + 5 * math.log2(case["nx"] * case["ny"]))}
    # forward, input gradient and weight gradient; weights, gradients and both moments in FP32
    flops, size = _gen_work(case["batch"])
    params = 1508864
    return {"bytes": case["iters"] * (size + params * 4.0 * 6), "flops": case["iters"] * 3.0 * flops}


# ---- the same in plain 64-bit torch -----------------------------------------------------
def _east(q):
    return torch.roll(q, -1, 2)


def _west(q):
    return torch.roll(q, 1, 2)


def _north(q):
    return torch.roll(q, -1, 1)


def _south(q):
    return torch.roll(q, 1, 1)


class _Exact:
    """The channel's time step on (nz + 2, ny, nx) arrays, periodic in x and y, one ghost
    plane per wall."""

    def __init__(self, nx, ny, nz, phys, u_crf=0.0):
        self.n = nx, ny, nz
        self.u_crf, self.force = u_crf, 1.0 - u_crf
        self.dxi, self.dyi, self.rei = nx / phys["lx"], ny / phys["ly"], 1.0 / phys["re"]
        h, _ = _mesh(nz, phys["lz"], phys["stretch_ratio"])
        self.h, self.hi = h[:, None, None], (1.0 / h)[:, None, None]
        self.ci = (2.0 / (h[:-1] + h[1:]))[:, None, None]  # 1 / distance of the centres k and k + 1
        self.weight = (h[1:-1] / phys["lz"])[:, None, None]
        # the wall-normal operator's reciprocal pivots for each pair of wavenumbers
        ex = 2.0 * (torch.cos(TWO_PI * torch.arange(nx // 2 + 1, dtype=torch.float64, device=DEVICE) / nx) - 1.0)
        ey = 2.0 * (torch.cos(TWO_PI * torch.arange(ny, dtype=torch.float64, device=DEVICE) / ny) - 1.0)
        lam = (ex * self.dxi ** 2)[None, :] + (ey * self.dyi ** 2)[:, None]
        up = (self.ci[1:-1] * self.hi[1:-2]).flatten().tolist() + [0.0]
        down = [0.0] + (self.ci[1:-1] * self.hi[2:-1]).flatten().tolist()
        self.down, self.up = down, up
        self.pivots = torch.empty((nz, ny, nx // 2 + 1), dtype=torch.float64, device=DEVICE)
        b = lam - up[0]
        for k in range(nz):
            if k:
                b = lam - (up[k] + down[k]) - down[k] * up[k - 1] * self.pivots[k - 1]
            self.pivots[k] = 1.0 / b
        self.pivots[nz - 1, 0, 0] = 0.0  # the free constant of the singular mode

    def bound(self, u, v, w):
        for q, wall in ((u, -self.u_crf), (v, 0.0)):
            q[0] = 2.0 * wall - q[1]
            q[-1] = 2.0 * wall - q[-2]
        w[0] = w[-2] = w[-1] = 0.0

    def start(self, fields):
        q = []
        for a in fields:
            nz, ny, nx = a.shape
            f = torch.zeros((nz + 2, ny, nx), dtype=torch.float64, device=DEVICE)
            f[1:-1] = a.double()
            q.append(f)
        q[0][1:-1] -= self.u_crf
        self.bound(*q)
        return q

    def rhs(self, u, v, w):
        """visc - conv of the three components on the interior planes."""
        dxi, dyi = self.dxi, self.dyi
        h0, hm, hp = self.h[1:-1], self.h[:-2], self.h[2:]
        hi0, hip = self.hi[1:-1], self.hi[2:]
        cm, c0 = self.ci[:-1], self.ci[1:]
        uc, vc, wc = u[1:-1], v[1:-1], w[1:-1]
        out = []
        # the values on the upper and lower faces of the cells of u and v
        up = [(q[1:-1] * hp + q[2:] * h0) * c0 for q in (u, v)]
        lo = [(q[1:-1] * hm + q[:-2] * h0) * cm for q in (u, v)]
        for c, q in ((0, u), (1, v)):
            qc = q[1:-1]
            e, wst = _east(qc), _west(qc)
            n, s = _north(qc), _south(qc)
            if c == 0:
                conv = ((qc + e) ** 2 - (wst + qc) ** 2) * dxi
                conv += ((qc + n) * (vc + _east(vc)) - (s + qc) * (_south(vc) + _south(_east(vc)))) * dyi
                wt = w[:-1] + _east(w[:-1])
            else:
                conv = ((uc + _north(uc)) * (qc + e) - (_west(uc) + _west(_north(uc))) * (wst + qc)) * dxi
                conv += ((qc + n) ** 2 - (s + qc) ** 2) * dyi
                wt = w[:-1] + _north(w[:-1])
            conv += (up[c] * wt[1:] - lo[c] * wt[:-1]) * hi0
            conv *= 0.25
            if self.u_crf:
                conv += 0.5 * self.u_crf * dxi * (e - wst)
            visc = (e - 2.0 * qc + wst) * dxi ** 2 + (n - 2.0 * qc + s) * dyi ** 2
            visc += ((q[2:] - qc) * c0 - (qc - q[:-2]) * cm) * hi0
            out.append(visc * self.rei - conv)
        e, wst, n, s = _east(wc), _west(wc), _north(wc), _south(wc)
        conv = (up[0] * (wc + e) - _west(up[0]) * (wst + wc)) * dxi
        conv += (up[1] * (wc + n) - _south(up[1]) * (s + wc)) * dyi
        conv += ((wc + w[2:]) ** 2 - (wc + w[:-2]) ** 2) * c0
        conv *= 0.25
        if self.u_crf:
            conv += 0.5 * self.u_crf * dxi * (e - wst)
        visc = (e - 2.0 * wc + wst) * dxi ** 2 + (n - 2.0 * wc + s) * dyi ** 2
        visc += ((w[2:] - wc) * hip - (wc - w[:-2]) * hi0) * c0
        out.append(visc * self.rei - conv)
        return out

    def project(self, u, v, w, dt):
        """Subtracts the gradient that makes the field divergence-free."""
        nx, ny, nz = self.n
        div = (u[1:-1] - _west(u[1:-1])) * self.dxi + (v[1:-1] - _south(v[1:-1])) * self.dyi
        div += (w[1:-1] - w[:-2]) * self.hi[1:-1]
        x = torch.fft.rfft2(div / dt)
        del div
        x[0] *= self.pivots[0]
        for k in range(1, nz):
            x[k] = (x[k] - self.down[k] * x[k - 1]) * self.pivots[k]
        for k in range(nz - 2, -1, -1):
            x[k] -= self.up[k] * self.pivots[k] * x[k + 1]
        p = torch.fft.irfft2(x, s=(ny, nx))
        del x
        u[1:-1] -= dt * self.dxi * (_east(p) - p)
        v[1:-1] -= dt * self.dyi * (_north(p) - p)
        w[1:-2] -= dt * (p[1:] - p[:-1]) * self.ci[1:-1]

    def step(self, q, dt):
        first = [torch.zeros_like(a) for a in q]
        for o, a, r in zip(first, q, self.rhs(*q)):
            o[1:-1] = a[1:-1] + dt * r
        self.bound(*first)
        for a, o, r in zip(q, first, self.rhs(*first)):
            a[1:-1] = (o[1:-1] + dt * r + a[1:-1]) * 0.5
        del first
        self.bound(*q)
        self.project(*q, dt)
        nx, ny, _ = self.n
        q[0][1:-1] += self.force - (q[0][1:-1] * self.weight).sum() / (nx * ny)
        self.bound(*q)

    def rate(self, q):
        u, v, w = q
        r = ((u[1:-1] + _west(u[1:-1])) * 0.5).abs() * self.dxi
        r += ((v[1:-1] + _south(v[1:-1])) * 0.5).abs() * self.dyi
        r += ((w[1:-1] + w[:-2]) * 0.5).abs() * self.hi[1:-1]
        return float(r.max())

    def steps(self, q, count, cfl, nt_check, after=None):
        dt = cfl / self.rate(q) if cfl > 0.0 else 2e-3
        for n in range(1, count + 1):
            self.step(q, dt)
            if cfl > 0.0 and (n % nt_check == 0 or n < nt_check and n & (n - 1) == 0):
                dt = cfl / self.rate(q)
            if after:
                after(n, q)


def _exact_step(case, seed):
    form = case.get("form", "fp64")
    phys = _physics(*_grid(case))
    ex = _Exact(*_grid(case), phys, case.get("u_crf", 0.0))
    q = ex.start(_start_fields(*_grid(case), phys, form, seed))
    sums = []

    def sample(n, q):
        if n % 10:
            return
        u, v, w = q
        u = (u[1:-1] + _west(u[1:-1])) * 0.5 + ex.u_crf
        v = (v[1:-1] + _south(v[1:-1])) * 0.5
        w = (w[1:-1] + w[:-2]) * 0.5
        sums.append(torch.stack([x.mean((1, 2)) for x in (u, v, w, u * u, v * v, w * w, u * v, u * w, v * w)]))

    ex.steps(q, case["steps"], case.get("cfl", 0.0), case["steps"], sample if case.get("stats") else None)
    out = {f: a[1:-1] for f, a in zip(FIELDS, q)}
    if case.get("stats"):
        out["stats"] = torch.stack(sums).mean(0)
    if case.get("judge"):
        u = q[0][1:-1] + ex.u_crf
        tau = [float((ex.rei * u[k] / (0.5 * ex.h[1])).mean()) for k in (0, -1)]
        re_tau = 0.5 * sum(math.sqrt(abs(t)) for t in tau) * 0.5 * phys["lz"] / ex.rei
        out["judged"] = torch.cat([u.mean((1, 2)), u.new_tensor([re_tau / 180.0])])
    return out


# the generator: latent, network, statistics, interpolation
def _splitmix(x):
    """SplitMix64's output for the counters x (numpy uint64, wrapping)."""
    x = x + np.uint64(0x9E3779B97F4A7C15)
    x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


def _word(x):
    return np.array([x & 0xFFFFFFFFFFFFFFFF], dtype=np.uint64)


def _latent(seed, shape):
    n = int(np.prod(shape))
    h1 = _splitmix(_word(seed * 0x100000001B3) + np.uint64(2) * np.arange(n, dtype=np.uint64))
    h2 = _splitmix(h1 ^ np.uint64(0xD1B54A32D192ED03))
    u1, u2 = (((h >> np.uint64(40)).astype(np.float64) + 0.5) / 16777216.0 for h in (h1, h2))
    z = np.sqrt(-2.0 * np.log(u1)) * np.cos(TWO_PI * u2)
    return torch.from_numpy(z.reshape(shape)).to(DEVICE)


def _conv(x, w):
    """3x3x3 convolution of (b, z, y, x, c), periodic in x and y, zero outside the walls."""
    y = None
    pad = torch.nn.functional.pad(x, (0, 0, 0, 0, 0, 0, 1, 1))
    for t in range(27):
        s = torch.roll(pad[:, t // 9:t // 9 + x.shape[1]], (1 - t // 3 % 3, 1 - t % 3), (2, 3))
        s = s @ w[t].T
        y = s if y is None else y + s
    return y


def _network(params, latent, r):
    """The generator's u, v, w at its cell centres; params as the flat vector."""
    at, x = 0, latent
    layers = _gen_layers()
    weights, films = [], []
    for ci, co, lv in layers:
        weights.append(params[at:at + 27 * ci * co].view(27, co, ci))
        at += 27 * ci * co
    for ci, co, lv in layers:
        nz = 64 >> (3 - lv)
        films.append(params[at:at + 4 * nz * co].view(4, nz, co))
        at += 4 * nz * co
    level = 0
    for i, ((ci, co, lv), w, f) in enumerate(zip(layers, weights, films)):
        if lv != level:
            for d in (1, 2, 3):
                x = x.repeat_interleave(2, d)
            level = lv
        rb = r[:, None, None]
        gam, bet = 1.0 + f[0] + f[1] * rb, f[2] + f[3] * rb
        x = gam[:, :, None, None] * _conv(x, w) + bet[:, :, None, None]
        if i + 1 < len(layers):
            x = torch.nn.functional.leaky_relu(x, 0.2)
    return x[..., :3]


def _plane_stats(f):
    """31 statistics of u, v, w per sample and plane: means, variances, the u-w covariance,
    covariances at lags of 1, 2, 4, 8 cells along x and y."""
    mu = f.mean((2, 3))
    s = [mu[..., c] for c in range(3)]
    s += [(f[..., c] ** 2).mean((2, 3)) - mu[..., c] ** 2 for c in range(3)]
    s.append((f[..., 0] * f[..., 2]).mean((2, 3)) - mu[..., 0] * mu[..., 2])
    for c in range(3):
        for d in (3, 2):
            for lag in (1, 2, 4, 8):
                s.append((f[..., c] * torch.roll(f[..., c], -lag, d)).mean((2, 3)) - mu[..., c] ** 2)
    return torch.stack(s, -1)


def _stored_params():
    bits = np.load(learned.WEIGHTS)["params_bf16"].astype(np.uint32) << 16
    return torch.from_numpy(bits.view(np.float32).astype(np.float64)).to(DEVICE)


def _exact_train(case, seed):
    d = np.load(learned.TARGETS)
    targets = torch.from_numpy(d["stats"]).to(DEVICE)
    re = d["re_tau"]
    batch, iters = case["batch"], case["iters"]
    scale = torch.full((31,), float(torch.sqrt((targets[..., 3] ** 2).mean())), dtype=torch.float64, device=DEVICE)
    scale[:3] = float(torch.sqrt((targets[..., 0] ** 2).mean()))
    p = _start_params(seed).double()
    m, v, losses = torch.zeros_like(p), torch.zeros_like(p), []
    seed &= 0xFFFF
    warm = min(100, iters // 10 + 1)
    for it in range(iters):
        rate = (it + 1.0) / warm if it < warm else 0.05 + 0.475 * (1.0 + math.cos(math.pi * (it - warm) / (iters - warm)))
        pick = _splitmix(_word((seed * 1000003 + it) * 0x9E3779B97F4A7C15) + np.arange(batch, dtype=np.uint64))
        t = (pick % np.uint64(len(re))).astype(np.int64)
        r = torch.from_numpy((re[t] - 260.0) / 140.0).to(DEVICE)
        q = p.clone().requires_grad_(True)
        z = _latent(seed * 7919 + 0x5BD1E995 * it, (batch, 8, 6, 8, 16))
        off = (_plane_stats(_network(q, z, r)) - targets[torch.from_numpy(t).to(DEVICE)]) / scale
        loss = (off ** 2).sum() / (batch * 64)
        loss.backward()
        losses.append(float(loss))
        m = 0.9 * m + 0.1 * q.grad
        v = 0.999 * v + 0.001 * q.grad ** 2
        p = p - 1e-3 * rate * (m / (1 - 0.9 ** (it + 1))) / (torch.sqrt(v / (1 - 0.999 ** (it + 1))) + 1e-8)
    return {"loss": torch.tensor(losses, dtype=torch.float64), "params": p}


def _exact_propose(case, seed):
    nx, ny, nz = _grid(case)
    r = torch.tensor([(case["re_tau"] - 260.0) / 140.0], dtype=torch.float64, device=DEVICE)
    f = _network(_stored_params(), _latent(seed & 0xFFFF, (1, 8, 6, 8, 16)), r)[0]
    phys = _physics(nx, ny, nz)
    ex = _Exact(nx, ny, nz, phys)
    h, zc = _mesh(nz, phys["lz"], phys["stretch_ratio"])
    zf = torch.cat([h.new_zeros(1), torch.cumsum(h[1:-1], 0)])
    zg = 0.5 * (zf[:-1:nz // 64] + zf[nz // 64::nz // 64])  # the generator's plane centres
    zg = torch.cat([zg.new_zeros(1), zg, zf[-1:]])
    planes = torch.nn.functional.pad(f, (0, 0, 0, 0, 0, 0, 1, 1))  # zero at the walls

    def along(a, at, dim):
        """Periodic linear interpolation of a at the cell coordinates `at` along dim."""
        n, lo = a.shape[dim], torch.floor(at)
        shape = [1] * a.dim()
        shape[dim] = -1
        t = (at - lo).view(shape)
        lo = lo.long() % n
        return (1.0 - t) * a.index_select(dim, lo) + t * a.index_select(dim, (lo + 1) % n)

    def place(c, x_off, y_off, z):
        k = torch.clamp(torch.searchsorted(zg, z) - 1, 0, 64)
        t = ((z - zg[k]) / (zg[k + 1] - zg[k])).view(-1, 1, 1)
        a = (1.0 - t) * planes[k, :, :, c] + t * planes[k + 1, :, :, c]
        i = (torch.arange(1, nx + 1, dtype=torch.float64, device=DEVICE) - x_off) * (64 / nx) - 0.5
        j = (torch.arange(1, ny + 1, dtype=torch.float64, device=DEVICE) - y_off) * (48 / ny) - 0.5
        return along(along(a, j, 1), i, 2)

    centres = 0.5 * (zf[1:] + zf[:-1])
    q = ex.start([place(0, 0.0, 0.5, centres), place(1, 0.5, 0.0, centres), place(2, 0.5, 0.5, zf[1:])])
    ex.project(*q, 2e-3)
    ex.bound(*q)
    return {name: a[1:-1] for name, a in zip(FIELDS, q)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "modules"):
        return _exact_step(case, seed)
    if kind == "propose":
        return _exact_propose(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    out = []
    for i, (nx, ny, nz, phys) in enumerate(_member_specs(case["specs"], case["members"])):
        ex = _Exact(nx, ny, nz, phys)
        q = ex.start(_start_fields(nx, ny, nz, phys, "mixed", 1000 * int(seed) + i))
        ex.steps(q, case["steps"], 0.5, case["steps"])
        out.append([a[1:-1] for a in q])
    return out
