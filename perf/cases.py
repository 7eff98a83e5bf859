"""The work that users of this framework have it do, as cases with inputs, one
pass through the public entry points, and the pass's result in 64 bits.

Kinds of case:
  step2d    one time step of a 2D Ti-Nb run (lib.Context.step) on a state from
            the middle of a run: frozen or coarse-grid temperature ("tfc": with
            the coarse grid's source and sub-steps, one whole turn of the
            loop), FP64 or FP32, exact CALPHAD or the trained network, with or
            without the per-step solute mass, with or without a moving-frame
            shift fused into the step.
  ensemble  steps of a batch of uneven runs (lib.Ensemble.steps).
  step3d    one time step of the 3D three-phase model (lib.Context3.step),
            TiAg or Ti-Nb CALPHAD energy, FP64 or FP32, exact or network.
  train     one minibatch step of the surrogate's training (gradient, Adam).
  tip       the output turn of the loop: coarse tip, precise tip, solute mass.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.abspath("2d-rapid-solidification_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from rapidsolid import _abi, configs, lib, surrogate  # noqa: E402

DEV = "cuda"


# ---------------------------------------------------------------- the cases

def _s2(nx, ny, precision, front, wave, **kw):
    """front: the front's mean column; wave: half the depth of its cells, in cells."""
    c = dict(kind="step2d", precision=precision, temperature="frozen", network=False, mass=False, nx=nx, ny=ny,
             front=front, wave=wave, G=5.0e6, V=0.5, noise=0.01, shift=0)
    c.update(kw)
    return c


def listed():
    return [
        # the reference's own small workload (Ti-10at%Nb, 256 x 256): a step is launch latency
        dict(_s2(256, 256, "f64", 16, 0.5, G=1.0e6, V=0.05, noise=0.0), name="f64_256"),
        # the drop-in precision at scale: planar front at column 16, melt ahead of it, interface noise
        dict(_s2(2048, 2048, "f64", 16, 0.5), name="f64_2048"),
        # the reference's default set-up (768 x 832, coarse-grid temperature, tip at Nx - 268) with a cellular front
        dict(_s2(768, 832, "f64", 500, 30.0, temperature="tfc", G=1.0e7, V=1.0, noise=0.0), name="f64_tfc_768x832"),
        # a domain of the user's own size: odd row length, front in mid-domain, grown cells behind it
        dict(_s2(1535, 1021, "f64", 700, 40.0, noise=0.0), name="f64_cells_1535x1021"),
        # the FP32 bulk run with its solute mass read every step
        dict(_s2(2048, 2048, "f32", 16, 0.5, mass=True), name="f32_2048"),
        # the same run through the trained network
        dict(_s2(2048, 2048, "f32", 16, 0.5, network=True), name="f32_network_2048"),
        # a parameter study: 16 uneven runs, 8 steps, their first moving-frame shift among them
        dict(kind="ensemble", runs=16, steps=8, smallest=256, largest_x=1024, largest_y=2048, sizes=2024,
             name="f32_ensemble_16"),
        # the 3D peritectic run, FP32 (512 x 512 columns; half of the 1024 planes)
        dict(kind="step3d", energy="tiag", precision="f32", network=False, nx=512, ny=512, nz=512, front=40, depth=6.0,
             name="f32_3d_512x512x512"),
        # the reference's own 3D extents, in its precision
        dict(kind="step3d", energy="tiag", precision="f64", network=False, nx=512, ny=512, nz=128, front=40, depth=6.0,
             name="f64_3d_512x512x128"),
        # the 3D Ti-Nb CALPHAD run of two grains
        dict(kind="step3d", energy="tinb", precision="f32", network=False, nx=512, ny=512, nz=256, front=24, depth=2.0,
             name="f32_3d_tinb_512x512x256"),
        # training the surrogate: the default minibatch
        dict(kind="train", batch=4096, name="train_4096"),
        # the tip, frame and mass figures of an output turn at scale
        dict(kind="tip", precision="f64", nx=2048, ny=2048, front=300, wave=40.0, name="tip_2048"),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step2d"] * 6 + ["step3d"] * 2 + ["ensemble", "train", "tip"])
    if kind == "step2d":
        while True:
            nx, ny = _size(rng, 128, 4096), _size(rng, 96, 4096)
            if nx * ny <= 9_000_000:
                break
        what = rng.choice(["f64", "f64", "tfc64", "f32", "f32", "tfc32", "network"])
        if rng.random() < 0.6:  # most programs round their extents
            nx, ny = (nx + 31) // 32 * 32, (ny + 31) // 32 * 32
        front = int(nx * rng.uniform(0.1, 0.7))
        wave = rng.choice([0.5, 0.5, rng.uniform(2.0, 0.08 * nx)])
        precision = "f64" if what.endswith("64") else "f32"
        if what.startswith("tfc"):
            ny = max(12, ny // 10) * 10 + 2  # the coarse grid holds whole blocks of 10 rows
            return _s2(nx, ny, precision, front, wave, temperature="tfc", G=1.0e7, V=1.0, noise=0.0)
        shift = rng.choice([0, 0, 0, rng.randint(-4, 12)])
        return _s2(nx, ny, precision, front, wave, network=what == "network", mass=rng.random() < 0.5,
                   V=rng.choice([0.05, 0.2, 0.5, 1.0]), noise=rng.choice([0.0, 0.01]), shift=shift)
    if kind == "step3d":
        e, p, n = rng.choice([("tiag", "f32", False), ("tiag", "f64", False), ("tinb", "f32", False),
                              ("tinb", "f64", False), ("tinb", "f32", True)])
        nx, ny, nz = _size(rng, 64, 384) // 4 * 4, _size(rng, 40, 384), _size(rng, 80, 400)
        return dict(kind="step3d", energy=e, precision=p, network=n, nx=nx, ny=ny, nz=nz,
                    front=int(nz * rng.uniform(0.15, 0.5)), depth=rng.uniform(0.5, 10.0))
    if kind == "ensemble":
        return dict(kind="ensemble", runs=rng.randint(4, 24), steps=rng.randint(3, 12), smallest=128, largest_x=768,
                    largest_y=1024, sizes=rng.randrange(1 << 30))
    if kind == "train":
        return dict(kind="train", batch=_size(rng, 500, 40000))
    nx, ny = _size(rng, 200, 4096), _size(rng, 128, 4096)
    return dict(kind="tip", precision=rng.choice(["f64", "f32"]), nx=nx, ny=ny, front=int(nx * rng.uniform(0.1, 0.6)),
                wave=rng.uniform(0.5, 0.05 * nx))


# ---------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform(g, *shape):
    return torch.rand(*shape, dtype=torch.float64, device=DEV, generator=g)


def _params2(case):
    """Run parameters of a 2D case: the Ti-10Nb workload, or the reference's defaults for the coarse-grid temperature."""
    if case.get("temperature") == "tfc":
        p = configs.default_params()
        p.nx_all, p.ny_all, p.i_tip_target = case["nx"], case["ny"], case["front"]
        return p
    p = configs.scale()
    p.nx_all, p.ny_all, p.i_tip_target = case["nx"], case["ny"], case["front"]
    p.GG, p.Vp = case.get("G", 5.0e6) * 1e-9, case.get("V", 0.5)
    p.noise_amplitude = case.get("noise", 0.0)
    return p


def _ghosts(f, periodic=True):
    f[1:-1, 0], f[1:-1, -1] = f[1:-1, 1], f[1:-1, -2]
    f[0], f[-1] = (f[-2], f[1]) if periodic else (f[1], f[-2])
    return f


def _state2(p, wave, g, solid, layer, tail):
    """psi and c in FP64: a front at i_tip_target whose cells are 2 wave deep (wave <= 1: the jitter of a planar
    front), the solid behind it, and ahead of it a solute layer of `layer` that decays over `tail` cells."""
    ny, nx = p.ny_all, p.nx_all
    j = torch.arange(ny, dtype=torch.float64, device=DEV)
    period = ny - 2
    if wave <= 1.0:
        i0 = p.i_tip_target + wave * (2.0 * _uniform(g, ny) - 1.0)
        steep = torch.ones_like(i0)
    else:
        n = max(1, round(period / max(24.0, 3.0 * wave)))  # cells along the front
        ph = 2.0 * math.pi * (_uniform(g, 2))
        w = 2.0 * math.pi * n / period
        u = torch.sin(w * j + ph[0])
        i0 = p.i_tip_target + wave * (u - 0.25 * torch.cos(2 * w * j + ph[1]))
        di = wave * w * (torch.cos(w * j + ph[0]) + 0.5 * torch.sin(2 * w * j + ph[1]))
        steep = torch.sqrt(1.0 + di * di)
    dist = (torch.arange(nx, dtype=torch.float64, device=DEV)[None, :] - i0[:, None]) / steep[:, None]
    psi = -torch.tanh(dist * p.dx / math.sqrt(2.0))
    h = 0.5 * (1.0 + psi)
    melt = p.cinf + layer * torch.exp(-dist.clamp_min(0.0) / tail)
    back = solid + 0.2 * layer * torch.sin(0.05 * dist + 6.0 * _uniform(g, ny)[:, None]).mul_(0.5)
    c = melt + (back - melt) * h
    return _ghosts(psi), _ghosts(c)


def _fill(fs, psi, c, p):
    fs.psi.copy_(psi)
    fs.c.copy_(c if fs.dtype == torch.float64 else c - p.cinf)


def _dtype(case):
    return torch.float64 if case["precision"] == "f64" else torch.float32


def _network(box, seed, target):
    """A network of the surrogate's shape fitted to `target` over the box: seeded hidden layers, a ridge fit of the
    last one (so a few 1e-3 of the targets' range, as a trained network has)."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1.0, 1.0, (8192, 3))
    y = target(0.5 * (box.T_lo + box.T_hi) + 0.5 * (box.T_hi - box.T_lo) * x[:, 0],
               0.5 * (box.c_lo + box.c_hi) + 0.5 * (box.c_hi - box.c_lo) * x[:, 1], x[:, 2])
    for q in range(2):
        box.y_mean[q], box.y_scale[q] = float(y[:, q].mean()), float(y[:, q].std())
    t = (y - y.mean(0)) / y.std(0)
    W1, b1 = rng.uniform(-1.5, 1.5, (32, 3)), rng.uniform(-1.0, 1.0, 32)
    W2, b2 = rng.uniform(-0.4, 0.4, (32, 32)), rng.uniform(-0.5, 0.5, 32)
    silu = lambda z: z / (1.0 + np.exp(-z))  # noqa: E731
    a = silu(silu(x @ W1.T + b1) @ W2.T + b2)
    A = np.concatenate([a, np.ones((len(a), 1))], 1)
    S = np.linalg.solve(A.T @ A + 1e-4 * len(a) * np.diag([1.0] * 32 + [0.0]), A.T @ t)
    w = np.concatenate([W1.ravel(), b1, W2.ravel(), b2, S[:32].T.ravel(), S[32]]).astype(np.float32)
    return torch.from_numpy(w).to(DEV), box


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.seed = case, seed
    return {"step2d": _prepare2, "ensemble": _prepare_ensemble, "step3d": _prepare3, "train": _prepare_train,
            "tip": _prepare_tip}[case["kind"]](s, case, _gen(seed))


def _prepare2(s, case, g):
    p = s.p = _params2(case)
    p.seed = s.seed
    s.ctx = lib.Context(p)
    s.cur, s.nxt = lib.FieldSet(p, _dtype(case)), lib.FieldSet(p, _dtype(case))
    if case["temperature"] == "tfc":
        d = s.ctx.d
        psi, c = _state2(p, case["wave"], g, 0.57, 0.07, 2.73)
        s.T = torch.zeros(d.NxT_all * d.NyT_all, dtype=torch.float64, device=DEV)
        s.ctx.temperature_init(s.T)
        T = s.T.view(d.NyT_all, d.NxT_all)[1:d.NyT - 1, 1:d.NxT - 1]  # the latent heat of the front's cells
        i = torch.arange(T.shape[1], dtype=torch.float64, device=DEV) - (p.i_tip_target + d.i_left_end_initial) / 10.0
        rows = torch.arange(T.shape[0], dtype=torch.float64, device=DEV)
        T += (0.4 + 0.1 * torch.sin(0.7 * rows + 6.0 * _uniform(g, 1)))[:, None] * torch.exp(-(i / 20.0) ** 2)
        whole = s.T.view(d.NyT_all, d.NxT_all)
        whole[0], whole[d.NyT - 1] = whole[d.NyT - 2].clone(), whole[1].clone()
        s.T2, s.source = torch.zeros_like(s.T), torch.zeros_like(s.T)
        s.step = 0
    else:
        D_over_V = p.Dl / p.Vp / (p.dx * p.S * p.W0)
        psi, c = _state2(p, case["wave"], g, 0.885, 0.015, D_over_V)
        s.step = 1000
        s.hist = 0
        s.l = s.step * p.Vp * s.ctx.d.dt * s.ctx.d.tau0 / (p.S * p.W0)
    _fill(s.cur, psi, c, p)
    s.mass = torch.zeros(1, dtype=torch.float64, device=DEV) if case["mass"] else None
    if case["network"]:
        s.w, s.box = _network(surrogate.fitted_box(), s.seed, lambda T, x, phi: _targets(p, T, x, _gg(phi)))
        s.ctx.set_surrogate(s.w, s.box)
    return s


def _prepare_ensemble(s, case, g):
    rng = np.random.default_rng(case["sizes"])
    s.params, s.sets = [], []
    for k in range(case["runs"]):
        p = configs.scale()
        p.nx_all = int(rng.integers(case["smallest"] // 4, case["largest_x"] // 4 + 1)) * 4
        p.ny_all = int(rng.integers(case["smallest"] // 4, case["largest_y"] // 4 + 1)) * 4
        p.Vp = float(np.exp(rng.uniform(np.log(0.05), np.log(2.0))))
        p.GG = float(np.exp(rng.uniform(np.log(1e5), np.log(1e7)))) * 1e-9
        p.i_tip_target, p.noise_amplitude, p.seed = 16, 0.0, s.seed + k
        s.params.append(p)
    s.ens = lib.Ensemble(s.params)
    for k, p in enumerate(s.params):
        a, b = lib.FieldSet(p, torch.float32), lib.FieldSet(p, torch.float32)
        _fill(a, *_state2(p, 0.5, g, 0.885, 0.015, p.Dl / p.Vp / (p.dx * p.S * p.W0)), p)
        s.ens.bind(k, a, b)
    return s


def _params3(case):
    make = configs.tinb_3d if case["energy"] == "tinb" else configs.peritectic_3d
    return make(nx=case["nx"], ny=case["ny"], nz=case["nz"])


def _prepare3(s, case, g):
    p = s.p = _params3(case)
    tinb = case["energy"] == "tinb"
    p.z_T = float(case["front"])
    s.ctx = lib.Context3(p)
    s.cur, s.nxt = lib.FieldSet3(p, _dtype(case)), lib.FieldSet3(p, _dtype(case))
    s.step = 10
    w = 2.0  # half width of the interfaces, in cells
    x = torch.arange(p.nx, dtype=torch.float64, device=DEV)[None, :]
    y = torch.arange(p.ny, dtype=torch.float64, device=DEV)[:, None]
    u = 2.0 * math.pi * _uniform(g, 4)
    kx, ky = 2.0 * math.pi / (p.nx - 2), 2.0 * math.pi / (p.ny - 2)
    zf = case["front"] + case["depth"] * torch.sin(3 * kx * x + u[0]) * torch.sin(2 * ky * y + u[1])
    # the second solid: lamellae along x (TiAg), one of two grains (Ti-Nb)
    n = 1 if tinb else 4
    lam = torch.sin(n * kx * x + u[2] + 0.3 * torch.sin(ky * y + u[3])) / (n * kx)
    share = 0.5 * (1.0 + torch.tanh(lam / w))
    if tinb:
        liquid, solid1, solid2, off = p.c_ref + 0.01, 0.885, 0.885, p.c_ref
    else:
        B1, B2 = p.B11 + p.B12 * p.T_ref, p.B21 + p.B22 * p.T_ref
        off = liquid = (B1 - 0.5 * B2) / (p.A1 - 0.5 * p.A2) + p.A1
        solid1 = (B1 + 0.5 * B2) / (p.A1 + 0.5 * p.A2) - p.A1 - p.A2
        solid2 = (B1 - 0.5 * B2) / (p.A1 - 0.5 * p.A2) - p.A1 + p.A2
    for z in range(1, p.nz - 1):
        h = 0.5 * (1.0 + torch.tanh((z - zf) / w))
        p2 = (1.0 - h) * share
        c = h * off + p2 * solid1 + (1.0 - h - p2) * solid2
        c += h * (liquid - off + (0.002 if not tinb else 0.0)) * torch.exp(-(z - zf).clamp_min(0.0) / 8.0)
        s.cur.phi1[z], s.cur.phi2[z] = h, p2
        s.cur.c[z] = c if s.cur.dtype == torch.float64 else c - off
    for f in (s.cur.phi1, s.cur.phi2, s.cur.c):
        _ghosts3(f)
    if case["network"]:
        q = configs.scale()
        q.cinf = p.c_ref
        s.w, s.box = _network(surrogate.fitted_box(), s.seed, lambda T, c, gv: _targets(q, T, c, gv))
        s.ctx.set_surrogate(s.w, s.box)
    return s


def _prepare_train(s, case, g):
    p = configs.scale()
    s.box = surrogate.default_box()
    n = case["batch"]
    s.x = (2.0 * _uniform(g, n, 3) - 1.0).float()
    X = s.x.double().cpu().numpy()
    b = s.box
    Y = _targets(p, 0.5 * (b.T_lo + b.T_hi) + 0.5 * (b.T_hi - b.T_lo) * X[:, 0],
                 0.5 * (b.c_lo + b.c_hi) + 0.5 * (b.c_hi - b.c_lo) * X[:, 1], _gg(X[:, 2]))
    s.y = torch.from_numpy(Y).float().to(DEV)
    for q in range(2):
        b.y_mean[q], b.y_scale[q] = float(Y[:, q].mean()), float(Y[:, q].std())
    s.w = torch.from_numpy(surrogate.init_weights(s.seed)).to(DEV)
    # a few epochs in: the moments are those of earlier minibatches
    s.m = 1e-2 * (2.0 * _uniform(g, s.w.numel()) - 1.0).float()
    s.v = (1e-4 + 1e-3 * _uniform(g, s.w.numel())).float()
    s.grad, s.loss = torch.zeros_like(s.w), torch.zeros(1, dtype=torch.float64, device=DEV)
    s.t, s.lr = 500, 3e-3
    return s


def _prepare_tip(s, case, g):
    p = s.p = _params2(case)
    s.ctx = lib.Context(p)
    s.cur = lib.FieldSet(p, _dtype(case))
    _fill(s.cur, *_state2(p, case["wave"], g, 0.885, 0.015, 4.1), p)
    s.itip = torch.zeros(1, dtype=torch.int32, device=DEV)
    s.tip = torch.zeros(C.sizeof(_abi.Tip), dtype=torch.uint8, device=DEV)
    s.mass = torch.zeros(1, dtype=torch.float64, device=DEV)
    return s


# ---------------------------------------------------------------- one pass

def run(s):
    case = s.case
    if case["kind"] == "step2d":
        if case["temperature"] == "tfc":
            ile = s.ctx.d.i_left_end_initial
            s.ctx.step(s.cur, s.nxt, s.step, T_coarse=s.T, i_left_end=ile, i_left_end_T=ile)
            s.ctx.integrate_phi(s.cur, s.nxt, s.source, ile)
            s.ctx.temperature_step(s.T, s.T2, s.source, s.step)
            s.cur, s.nxt = s.nxt, s.cur
            s.step += 1
            d = s.ctx.d
            return s.cur.psi, s.cur.c, s.T.view(d.NyT_all, d.NxT_all)[:d.NyT, :d.NxT]  # without its padding
        s.ctx.step(s.cur, s.nxt, s.step, i_offset_history=s.hist + case["shift"], l_offset_Vp=s.l,
                   pull_back=case["shift"] or None, mass_out=s.mass)
        return (s.nxt.psi, s.nxt.c) if s.mass is None else (s.nxt.psi, s.nxt.c, s.mass)
    if case["kind"] == "ensemble":
        s.ens.steps(case["steps"])
        sets = [s.ens.state(k)[3] for k in range(case["runs"])]
        return [f.psi for f in sets], [f.c for f in sets]
    if case["kind"] == "step3d":
        s.ctx.step(s.cur, s.nxt, s.step)
        return s.nxt.phi1, s.nxt.phi2, s.nxt.c
    if case["kind"] == "train":
        L, st = s.ctx_lib(), lib._stream(None)
        s.grad.zero_()
        s.loss.zero_()
        n = case["batch"]
        lib.check(L.rs_mlp_grad(C.byref(s.box), lib._ptr(s.w), n, lib._ptr(s.x), lib._ptr(s.y), lib._ptr(s.grad),
                                lib._ptr(s.loss), st))
        s.t += 1
        lib.check(L.rs_mlp_adam(lib._ptr(s.w), lib._ptr(s.grad), lib._ptr(s.m), lib._ptr(s.v), s.t, s.lr, 1.0 / n, st))
        return s.grad, s.loss, s.w, s.m, s.v
    s.ctx.itip(s.cur, s.itip)
    s.ctx.precise_tip(s.cur, s.tip)
    s.ctx.mass(s.cur, s.mass)
    return s.itip, s.tip[:12].view(torch.int32), s.tip[16:].view(torch.float64), s.mass


_State.ctx_lib = staticmethod(lib.load)


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        rng = np.random.default_rng(case["sizes"])
        cells = 0
        for _ in range(case["runs"]):
            cells += 16 * int(rng.integers(case["smallest"] // 4, case["largest_x"] // 4 + 1)) * int(
                rng.integers(case["smallest"] // 4, case["largest_y"] // 4 + 1))
            rng.uniform(), rng.uniform()
        return {"bytes": 16.0 * cells * case["steps"], "flops": 60.0 * cells * case["steps"]}
    if kind == "train":
        n = case["batch"]
        return {"bytes": 20.0 * n + 7 * 4.0 * 1250, "flops": 6.0 * 1184 * n}
    size = 8 if case["precision"] == "f64" else 4
    cells = float(case["nx"] * case["ny"])
    if kind == "step2d":
        nbytes = 4 * size * cells
        if case["temperature"] == "tfc":  # psi twice for the source, the coarse grid's three arrays
            nT = (6667 + 61) // 64 * 64 * ((case["ny"] - 2) // 10 + 2)
            nbytes += 2 * size * cells + 4 * 8 * nT
        return {"bytes": nbytes, "flops": 60.0 * cells}
    if kind == "step3d":
        return {"bytes": 6 * size * cells * case["nz"], "flops": 80.0 * cells * case["nz"]}
    return {"bytes": 2 * size * cells, "flops": 2.0 * cells}


# ---------------------------------------------------------------- 64-bit results
# Plain torch (numpy for the network's fit) in FP64: the model's equations as
# they are written, on a backend-neutral `where`/`log`, no kernel of the framework.

L0_BCC, L0_LIQ = 12315.25, 5144.29


def _gibbs(T):
    """The pure elements' Gibbs energies at T: Ti BCC, Ti liquid, Nb BCC, Nb liquid (SGTE, 1300 K <= T < 2750 K)."""
    m = torch if isinstance(T, torch.Tensor) else np
    TlT = T * m.log(T)
    low, iT = T < 1941.0, 1.0 / T
    tb = m.where(low, 6667.385 + 105.366379 * T - 22.3771 * TlT + 1.21707e-3 * T**2 - 0.84534e-6 * T**3 - 2002750.0 * iT,
                 26483.26 - 182.426471 * T + 19.0900905 * TlT - 22.00832e-3 * T**2 + 1.228863e-6 * T**3
                 + 1400501.0 * iT)
    tl = m.where(low, 369519.198 - 2554.0225 * T + 342.059267 * TlT - 163.409355e-3 * T**2 + 12.457117e-6 * T**3
                 - 67034516.0 * iT, -19887.066 + 298.7367 * T - 46.29 * TlT)
    nb = -8519.353 + 142.045475 * T - 26.4711 * TlT + 0.203475e-3 * T**2 - 0.35012e-6 * T**3 + 93399.0 * iT
    return tb, tl, nb, nb + 29781.555 - 10.816418 * T - 306.098e-25 * T**7


def _gg(p):
    return 1.875 * p - 1.25 * p**3 + 0.375 * p**5


def _drive(T, c):
    """Gl - Gs (the ideal mixing terms are the same)."""
    tb, tl, nb, nl = _gibbs(T)
    return (1.0 - c) * (nl - nb) + c * (tl - tb) + c * (1.0 - c) * (L0_LIQ - L0_BCC)


def _mu(T, c, gS, RR):
    """Chemical potential at solid weight gS."""
    m = torch if isinstance(c, torch.Tensor) else np
    tb, tl, nb, nl = _gibbs(T)
    return gS * (tb - nb + L0_BCC * (1.0 - 2.0 * c)) + (1.0 - gS) * (tl - nl + L0_LIQ * (1.0 - 2.0 * c)) \
        + RR * T * m.log(c / (1.0 - c))


def _mu_melt(T, cinf, RR):
    """The melt's chemical potential at its nominal composition, the reference of the network's first output."""
    return _mu(T, np.float64(cinf) if not isinstance(T, torch.Tensor) else torch.full_like(T, cinf), 0.0, RR)


def _targets(p, T, c, g):
    return np.stack([_mu(T, c, 0.5 * (1.0 + g), p.RR) - _mu_melt(T, p.cinf, p.RR), _drive(T, c)], 1)


def _net(s, T, c, third):
    """The network in 64 bits (torch): its two outputs, unscaled."""
    b = s.box
    w = s.w.double()
    W1, b1 = w[:96].view(32, 3), w[96:128]
    W2, b2 = w[128:1152].view(32, 32), w[1152:1184]
    W3, b3 = w[1184:1248].view(2, 32), w[1248:]
    x = torch.stack([(T - 0.5 * (b.T_lo + b.T_hi)) / (0.5 * (b.T_hi - b.T_lo)),
                     (c - 0.5 * (b.c_lo + b.c_hi)) / (0.5 * (b.c_hi - b.c_lo)), third], -1)
    silu = torch.nn.functional.silu
    o = silu(silu(x @ W1.T + b1) @ W2.T + b2) @ W3.T + b3
    return [b.y_mean[q] + b.y_scale[q] * o[..., q] for q in (0, 1)]


def _philox(cell, step, seed):
    """Philox4x32-10 words of (cell, step) under the seed, as int64 tensors."""
    M = 0xFFFFFFFF
    x = [cell & M, cell >> 32, torch.full_like(cell, step & M), torch.full_like(cell, (step >> 32) ^ 0x4E4F4953)]
    k0, k1 = seed & M, seed >> 32
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
        p0, p1 = 0xD2511F53 * x[0], 0xCD9E8D57 * x[2]
        x = [(p1 >> 32 & M) ^ x[1] ^ k0, p1 & M, (p0 >> 32 & M) ^ x[3] ^ k1, p0 & M]
    return x


def _noise(cell, step, seed):
    a, b, c, d = _philox(cell, step, seed)
    u = lambda h, l: ((h >> 5).double() * 67108864.0 + (l >> 6).double() + 0.5) / 9007199254740992.0  # noqa: E731
    return torch.sqrt(-2.0 * torch.log(u(a, b))) * torch.cos(2.0 * math.pi * u(c, d))


def _derived(p):
    tau0 = (p.S * p.W0) ** 2 / (p.Gamma * p.muk0)
    dt = p.dt
    if dt <= 0:
        dt = 0.6 * p.dx * p.dx / 4.0 / max(1.0, p.Dl * tau0 / (p.S * p.W0) ** 2)
    latent = p.latent_heat * p.num_moles
    hh = p.Gamma * 1e-9 * latent / p.Tmelt / (2.0 * math.sqrt(2.0) / 3.0 * p.S * p.W0 * 1e-9)
    return tau0, dt, hh, p.RR * p.Tmelt / p.v0


def _shift2(p, psi, c, k):
    """The moving frame: columns move back by k."""
    i = (torch.arange(p.nx_all, device=DEV) + k).clamp(1, p.nx_all - 2)
    c = c[:, i].clone()
    c[:, i == p.nx_all - 2] = p.cinf
    return psi[:, i].clone(), c


def _step2(p, psi, c, T, step, net=None):
    """One time step of (psi, c) at the temperature T (a row of columns, or a field)."""
    tau0, dt, hh, h0 = _derived(p)
    phi, dx = psi.clamp(-1.0, 1.0), p.dx

    def at(f, a, b):  # the interior's neighbour at (i + a, j + b)
        return f[1 + b:f.shape[0] - 1 + b, 1 + a:f.shape[1] - 1 + a]
    ce, ea, we, no, so = at(phi, 0, 0), at(phi, 1, 0), at(phi, -1, 0), at(phi, 0, 1), at(phi, 0, -1)
    ne, nw, se, sw = at(phi, 1, 1), at(phi, -1, 1), at(phi, 1, -1), at(phi, -1, -1)
    px, py = (ea - we) / (2 * dx), (no - so) / (2 * dx)
    pxx, pyy, pxy = (ea - 2 * ce + we) / dx**2, (no - 2 * ce + so) / dx**2, (ne - nw - se + sw) / (4 * dx**2)
    lap = 2 / 3 * (pxx + pyy) + (ne + nw + se + sw - 4 * ce) / (6 * dx**2)
    g2 = px * px + py * py
    ok = torch.sqrt(g2) > 1e-15
    s2 = torch.where(ok, g2, torch.ones_like(g2))
    zero = torch.zeros_like(g2)
    tx, ty = (torch.where(ok, v, zero) for v in ((px * pxy - py * pxx) / s2, (px * pyy - py * pxy) / s2))
    cs, sn = (torch.where(ok, v / torch.sqrt(s2), zero) for v in (px, py))
    n4 = cs**4 + sn**4
    d1 = 4 * cs * sn * (sn**2 - cs**2)
    d2 = 4 * (6 * cs**2 * sn**2 - cs**4 - sn**4)
    a_s, a_k = 1 - 3 * p.eps1 + 4 * p.eps1 * n4, 1 - 3 * p.epk1 + 4 * p.epk1 * n4
    da1, da2 = 4 * p.eps1 * d1, 4 * p.eps1 * d2
    aniso = a_s**2 * lap + 2 * a_s * da1 * (tx * px + ty * py) + (da2 * a_s + da1**2) * (ty * px - tx * py)
    T = T.expand(c.shape)
    dG, gS = _drive(T, c), 0.5 * (1.0 + _gg(psi))
    mu = _mu(T, c, gS, p.RR)
    if net is not None:  # the network stands in for the cells outside the melt
        nm, nd = net(T, c, psi)
        melt = psi == -1.0
        mu = torch.where(melt, mu, nm + _mu_melt(T, p.cinf, p.RR))
        dG = torch.where(melt, dG, nd)
    term = ce - ce**3 + aniso + at(dG, 0, 0) * 1.875 * (1 - ce**2) ** 2 / (2 * hh * p.v0)
    new = ce + dt * a_k / a_s**2 * term
    if p.noise_amplitude > 0:
        jj, ii = torch.nonzero(1 - ce**2 > 1e-3, as_tuple=True)
        cell = (jj + 1) * p.nx_all + ii + 1
        new[jj, ii] += p.noise_amplitude * math.sqrt(dt) * (1 - ce[jj, ii] ** 2) * _noise(cell, step, p.seed)
    psi2, c2 = psi.clone(), c.clone()
    psi2[1:-1, 1:-1] = new.clamp_max(1.0)
    S = (0.5 * p.AA * (1 - psi) - 0.25 * (p.AA - 1) * (1 - psi) ** 2) * c * (1 - c)
    flux = 0.0
    for a, b in ((1, 0), (-1, 0), (0, 1), (0, -1)):
        side = [(a, 1), (a, -1), (0, 1), (0, -1)] if b == 0 else [(1, b), (-1, b), (1, 0), (-1, 0)]
        weight = 1.5 * (at(S, a, b) + at(S, 0, 0)) + 0.25 * sum(at(S, *q) for q in side)
        flux = flux + 0.25 * weight * (at(mu, a, b) - at(mu, 0, 0))
    c2[1:-1, 1:-1] = (at(c, 0, 0) + dt * p.Dl / (p.Gamma * p.muk0) / (h0 * p.v0) * flux / dx**2).clamp_min(1e-6)
    return _ghosts(psi2), _ghosts(c2)


def _frozen(p, hist, l):
    i = torch.arange(p.nx_all, dtype=torch.float64, device=DEV)
    dT0 = p.Tmelt - p.T_ref
    delta = p.delta_initial + p.GG * (i - p.i_tip_target + hist) * p.dx * p.S * p.W0 / dT0 - p.GG * l * p.S * p.W0 / dT0
    return (delta * dT0 + p.Tmelt)[None, :]


def _read2(fs, p):
    return fs.psi.double(), fs.c.double() + (0.0 if fs.dtype == torch.float64 else p.cinf)


def _exact2(s, case):
    p = s.p
    psi, c = _read2(s.cur, p)
    off = 0.0 if s.cur.dtype == torch.float64 else p.cinf
    if case["temperature"] == "tfc":
        d, r = s.ctx.d, p.ratio_dxT_dx
        tau0, dt, _, _ = _derived(p)
        T = s.T.view(d.NyT_all, d.NxT_all).clone()
        i = torch.arange(p.nx_all, device=DEV) - 1 + d.i_left_end_initial
        j = torch.arange(p.ny_all, device=DEV).double() - 1 + p.dx * r
        iT, jT = i // r, (j / r).long()
        x, y = (i.double() / r - iT)[None, :], (j / r - jT)[:, None]
        f = [T[jT + b][:, iT + a] for a, b in ((0, 0), (1, 0), (0, 1), (1, 1))]
        fine = f[0] + (f[1] - f[0]) * x + (f[2] - f[0]) * y + (f[3] - f[1] - f[2] + f[0]) * x * y
        psi2, c2 = _step2(p, psi, c, fine, s.step)
        src = torch.zeros_like(T)
        diff = (psi2 - psi)[1:-1, 1:-1]
        rows = diff.reshape(diff.shape[0] // r, r, -1).sum(1)
        src[1:1 + rows.shape[0]] = 0.5 * torch.zeros_like(src[1:1 + rows.shape[0]]).index_add_(1, i[1:-1] // r, rows)
        h = p.dx * r
        a = T[1:d.NyT - 1, 1:d.NxT - 1]
        ea, we = T[1:d.NyT - 1, 2:d.NxT], T[1:d.NyT - 1, :d.NxT - 2]
        no, so = T[2:d.NyT, 1:d.NxT - 1], T[:d.NyT - 2, 1:d.NxT - 1]
        rate = p.Vp * tau0 / (p.S * p.W0) * (ea - we) / (2 * h) + (ea + we + no + so - 4 * a) / h**2 * p.DT / (p.Gamma * p.muk0)
        assert d.ratio_dt_dtT == 1
        T2 = T.clone()
        T2[1:d.NyT - 1, 1:d.NxT - 1] = a + dt * rate + p.latent_heat / p.cp * src[1:d.NyT - 1, 1:d.NxT - 1] / r**2
        # the border of the coarse grid is held or copied
        length = math.ceil(p.length_sample_um * 1000 / (p.dx * p.S * p.W0 * r)) * (p.dx * p.S * p.W0 * r)
        T2[:, 0], T2[:, d.NxT - 1] = p.Tcold, p.Tcold + p.GG * length
        T2[0], T2[d.NyT - 1] = T2[d.NyT - 2].clone(), T2[1].clone()
        return psi2, c2 - off, T2[:d.NyT, :d.NxT]
    if case["shift"]:
        psi, c = _shift2(p, psi, c, case["shift"])
    net = (lambda T, x, phi: _net(s, T, x, phi)) if case["network"] else None
    psi2, c2 = _step2(p, psi, c, _frozen(p, s.hist + case["shift"], s.l), s.step, net)
    out = (psi2, c2 - off)
    return out if s.mass is None else out + (c2[1:-1, 1:-1].sum().reshape(1),)


def _itip(psi):
    cols = torch.nonzero((psi > 0).any(0)).flatten()
    return max(1, int(cols[-1])) if cols.numel() else 1


def _exact_ensemble(s, case):
    out = [], []
    for k, p in enumerate(s.params):
        psi, c = _read2(s.ens.sets[k][0], p)
        tau0, dt, _, _ = _derived(p)
        cadence = int(p.S * p.W0 * p.dx / (p.Vp * dt * tau0))
        hist, l = 0, 0.0
        for n in range(case["steps"]):
            if n % cadence == 0:
                k0 = _itip(psi) - p.i_tip_target
                hist += k0
                psi, c = _shift2(p, psi, c, k0)
            psi, c = _step2(p, psi, c, _frozen(p, hist, l), n)
            l += p.Vp * dt * tau0 / (p.S * p.W0)
        out[0].append(psi)
        out[1].append(c - p.cinf)
    return out


def _ghosts3(f):
    f[:, :, 0], f[:, :, -1] = f[:, :, -2], f[:, :, 1]
    f[:, 0], f[:, -1] = f[:, -2].clone(), f[:, 1].clone()
    f[0], f[-1] = f[1], f[-2]
    return f


def _step3(p, p1, p2, c, z0, step, net):
    """phi1, phi2 and c of the interior planes of a slab (its first and last plane are neighbours; z0: the first's index)."""
    tinb = p.energy == 1
    p3 = 1.0 - p1 - p2
    z = (torch.arange(c.shape[0], dtype=torch.float64, device=DEV) + z0)
    gi = lambda a, b, d: a * a * 0.25 * (15 * (1 - a) * (1 + a - (d - b) ** 2) + a * (9 * a * a - 5))  # noqa: E731
    g1 = lambda a, b, d: 3.75 * a * (2 - a - 4 * a * a + 3 * a**3 + (3 * a - 2) * (b - d) ** 2)  # noqa: E731
    g2 = lambda a, b, d: 7.5 * (a - 1) * a * a * (b - d)  # noqa: E731
    shape = (-1, 1, 1)
    if tinb:
        zi = z.clamp(1, p.nz - 2)  # ghost planes are images
        T = (p.T_ref + p.G_T * (zi - p.z_T - p.V_T * step)).view(shape).expand(c.shape)
        liquid = gi(p1, p2, p3)
        mu, dG = _mu(T, c, 1.0 - liquid, p.RR), _drive(T, c)
        if net is not None:
            melt = (p1 == 1.0) & (p2 == 0.0)
            nm, nd = net(T, c, 1.0 - 2.0 * liquid)
            mu = torch.where(melt, mu, nm + _mu_melt(T, p.c_ref, p.RR))
            dG = torch.where(melt, dG, nd)
        S = (p1 * (p.AA - (p.AA - 1) * p1) + p.Da * p2 + p.Db * p3) * c * (1 - c)
    else:
        r = (p.A1, -p.A1 - p.A2, -p.A1 + p.A2)
        mu = c - r[0] * gi(p1, p2, p3) - r[1] * gi(p2, p3, p1) - r[2] * gi(p3, p1, p2)
        T = p.T_ref + (p.G_T * (z - p.z_T - p.V_T * step) if p.G_T else 0.0 * z)
        B1, B2 = (p.B11 + p.B12 * T).view(shape), (p.B21 + p.B22 * T).view(shape)
        S = p1 + p.Da * p2 + p.Db * p3

    def at(f, a=0, b=0, d=0):
        n = f.shape
        return f[1 + d:n[0] - 1 + d, 1 + b:n[1] - 1 + b, 1 + a:n[2] - 1 + a]
    q1, q2, q3, m = at(p1), at(p2), at(p3), at(mu)
    if tinb:
        w = at(dG)
        f1, f2, f3 = g1(q1, q2, q3) * w, g2(q1, q2, q3) * w, g2(q1, q3, q2) * w
    else:
        e1, e2, e3 = (B1[1:-1] - r[0] * m), (-B1 - B2)[1:-1] - r[1] * m, (B2 - B1)[1:-1] - r[2] * m
        f1 = g1(q1, q2, q3) * e1 + g2(q2, q1, q3) * e2 + g2(q3, q1, q2) * e3
        f2 = g2(q1, q2, q3) * e1 + g1(q2, q3, q1) * e2 + g2(q3, q2, q1) * e3
        f3 = g2(q1, q3, q2) * e1 + g2(q2, q3, q1) * e2 + g1(q3, q1, q2) * e3
    ax = (((1, 0, 0), p.dx_inv), ((0, 1, 0), p.dy_inv), ((0, 0, 1), p.dz_inv))
    lap = lambda f: sum((at(f, *o) + at(f, *(-k for k in o)) - 2 * at(f)) * h * h for o, h in ax)  # noqa: E731
    l1, l2 = lap(p1), lap(p2)
    l3, b = -l1 - l2, p.b
    w1 = 2 * q1 * (1 - q1) * (1 - 2 * q1) + p.a1 * (q2 * q3) ** 2 * (3 + 2 * b * q1) \
        + 2 * p.a2 * q1 * q3**2 * (3 * q1 * q3 + 3 * q2 + b * q2**2) \
        + 2 * p.a3 * q1 * q2**2 * (3 * q1 * q2 + 3 * q3 + b * q3**2) + p.lam * f1 - l1
    w2 = 2 * q2 * (1 - q2) * (1 - 2 * q2) + 2 * p.a1 * q2 * q3**2 * (3 * q2 * q3 + 3 * q1 + b * q1**2) \
        + p.a2 * (q1 * q3) ** 2 * (3 + 2 * b * q2) + 2 * p.a3 * q2 * q1**2 * (3 * q1 * q2 + 3 * q3 + b * q3**2) \
        + p.lam * f2 - l2
    w3 = 2 * q3 * (1 - q3) * (1 - 2 * q3) + 2 * p.a1 * q3 * q2**2 * (3 * q2 * q3 + 3 * q1 + b * q1**2) \
        + 2 * p.a2 * q3 * q1**2 * (3 * q1 * q3 + 3 * q2 + b * q2**2) + p.a3 * (q1 * q2) ** 2 * (3 + 2 * b * q3) \
        + p.lam * f3 - l3
    flux = 0.0
    for o, h in ax:
        for sgn in (1, -1):
            k = tuple(sgn * v for v in o)
            flux = flux + 0.5 * (at(S, *k) + at(S)) * (at(mu, *k) - m) * h * h
    return (q1 - p.dt * (2 * w1 - w2 - w3) / 3, q2 - p.dt * (2 * w2 - w1 - w3) / 3, at(c) + p.dt * p.alpha * flux)


def _exact3(s, case):
    p, f32 = s.p, s.cur.dtype == torch.float32
    off = 0.0
    if f32:
        B1, B2 = p.B11 + p.B12 * p.T_ref, p.B21 + p.B22 * p.T_ref
        off = p.c_ref if p.energy == 1 else (B1 - 0.5 * B2) / (p.A1 - 0.5 * p.A2) + p.A1
    net = (lambda T, c, third: _net(s, T, c, third)) if case["network"] else None
    out = [torch.zeros(p.nz, p.ny, p.nx, dtype=torch.float64, device=DEV) for _ in range(3)]
    n = max(1, 8_000_000 // (p.nx * p.ny))
    for z in range(1, p.nz - 1, n):
        e = min(p.nz - 1, z + n)
        a, b, c = (f[z - 1:e + 1].double() for f in (s.cur.phi1, s.cur.phi2, s.cur.c))
        for o, v in zip(out, _step3(p, a, b, c + off, z - 1, s.step, net)):
            o[z:e, 1:-1, 1:-1] = v
    out[2] -= off
    return tuple(_ghosts3(o) for o in out)


def _exact_train(s, case):
    w = s.w.double().requires_grad_()
    W1, b1, W2, b2 = w[:96].view(32, 3), w[96:128], w[128:1152].view(32, 32), w[1152:1184]
    W3, b3 = w[1184:1248].view(2, 32), w[1248:]
    silu = torch.nn.functional.silu
    mean, scale = (torch.tensor(list(v), dtype=torch.float64, device=DEV) for v in (s.box.y_mean, s.box.y_scale))
    o = silu(silu(s.x.double() @ W1.T + b1) @ W2.T + b2) @ W3.T + b3
    loss = ((o - (s.y.double() - mean) / scale) ** 2).sum()
    loss.backward()
    g = w.grad / case["batch"]
    m, v, t = 0.9 * s.m.double() + 0.1 * g, 0.999 * s.v.double() + 0.001 * g * g, s.t + 1
    w2 = w.detach() - s.lr * (m / (1 - 0.9**t)) / (torch.sqrt(v / (1 - 0.999**t)) + 1e-8)
    return w.grad, loss.detach().reshape(1), w2, m, v


def _exact_tip(s, case):
    p = s.p
    psi = s.cur.psi.double().cpu().numpy()
    c = s.cur.c.double() + (0.0 if s.cur.dtype == torch.float64 else p.cinf)
    mass = c[1:-1, 1:-1].sum().reshape(1)
    last = np.where((psi[:, :-1] > 0).any(1), psi.shape[1] - 2 - np.argmax(psi[:, -2::-1] > 0, 1), 0)
    best, tj = 0.0, 0
    for j in range(p.ny_all):  # the row whose crossing reaches furthest
        i0 = int(last[j]) if last[j] >= int(best) else 0
        at = i0 + (psi[j, i0 + 1] - psi[j, i0]) * (0.0 - psi[j, i0])
        if at > best:
            best, tj = at, j
    xs, ys = [], []
    for j in range(tj - 2, tj + 3):
        j0 = j + (p.ny_all - 2 if j < 1 else -(p.ny_all - 2) if j > p.ny_all - 2 else 0)
        i = np.arange(last[j0] - 2, last[j0] + 3)
        y = psi[j0, i]
        # the quartic through five points of the profile, at psi = 0
        xs.append(sum(i[a] * np.prod([(0.0 - y[b]) / (y[a] - y[b]) for b in range(5) if b != a]) for a in range(5)))
        ys.append(float(j0))
    M = np.stack([np.ones(5), np.array(ys), np.array(ys) ** 2], 1)
    a0, a1, a2 = np.linalg.solve(M.T @ M, M.T @ np.array(xs))
    R = min(max(abs(1.0 / (2.0 * a2)) * p.dx * p.W0 * p.S, 1.0), 1e5)
    y0 = -a1 / (2.0 * a2)
    fit = torch.tensor([a0 - a2 * y0 * y0, y0, R], dtype=torch.float64)
    return None, None, fit, mass


def exact(case, seed):
    s = prepare(case, seed)
    return {"step2d": _exact2, "ensemble": _exact_ensemble, "step3d": _exact3, "train": _exact_train,
            "tip": _exact_tip}[case["kind"]](s, case)
