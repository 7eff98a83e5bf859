"""The forms of a 2D tile (far melt, deep solid, and the phases for every other
tile) and the tile heights, against the oracle: grids on both sides of every
line of the height rule, last tiles of one row and of all rows, last columns of
2 and 64 cells, fields of all melt, all solid, melt with solute up to and over
the far-melt bound, and a front with solid behind it and melt ahead; noise on,
so that listed cells are of both kinds.  Tolerances as in the single-step tests
of test_gpu_step.py (the same arithmetic on the same cells)."""
import numpy as np
import pytest

import pyoracle
from helpers import fix_ghosts, maxabs
from rapidsolid import configs, lib
from test_gpu_step import download, upload

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def state(p, kind, seed):
    rng = np.random.default_rng(seed)
    s = pyoracle.initial_planar(p, configs.C_LIQUID_TI10NB, configs.C_SOLID_AT_TLIQ, seed)
    ny, nx = s.psi.shape
    tiny = 1e-3 * min(p.cinf, 1 - p.cinf)
    if kind == "melt":
        s.psi[:] = -1.0
        s.c[:] = p.cinf + 0.9 * tiny * (2 * rng.random((ny, nx)) - 1)
    elif kind == "layer":  # some tiles far melt, some over its bound by a little or a lot
        s.psi[:] = -1.0
        s.c[:] = p.cinf + tiny * np.exp(2.0 * np.sin(np.arange(nx) / 40.0))[None, :] * (2 * rng.random((ny, nx)) - 1)
    elif kind == "solid":
        s.psi[:] = 1.0
        s.c[:] = 0.88 + 0.01 * rng.random((ny, nx))
    else:  # front: cells of the front, solid and melt on both sides
        i0 = p.i_tip_target + 20 * np.sin(2 * np.pi * 3 * np.arange(ny) / (ny - 2))
        s.psi[:] = -np.tanh((np.arange(nx)[None, :] - i0[:, None]) * p.dx / np.sqrt(2.0))
        s.c[:] = p.cinf + (0.88 - p.cinf) * 0.5 * (1 + s.psi) + 1e-4 * (1 - s.psi**2) * rng.standard_normal((ny, nx))
    s.phi[:] = s.psi
    fix_ghosts(p, s)
    return s


# FP64 tiles of 64 columns: 4 rows below one wave of 740 16-row tiles, 8 below three, then 16; FP32 tiles of
# 128: 4 below one, 8 below two
SIZES = [(64, 18), (128, 19), (260, 8), (320, 66), (2048, 371), (2052, 372), (2048, 1127), (2112, 1045), (2048, 1500)]


# rows that are not 16-byte aligned: a last tile column of one cell more or less than full, of the ghost column alone
ODD_SIZES = [(63, 18), (65, 19), (66, 20), (129, 66), (131, 22), (257, 40), (2047, 371), (2049, 372), (2049, 1127),
             (2111, 1045)]


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("kind", ["melt", "layer", "solid", "front"])
@pytest.mark.parametrize("nx,ny", SIZES + ODD_SIZES)
def test_tile_forms_match_the_oracle(nx, ny, kind, dtype):
    p = configs.small(nx, ny, i_tip_target=nx // 2, G=5e6, V=0.5, noise_amplitude=0.02, seed=9)
    d = pyoracle.derive(p)
    s = state(p, kind, nx + ny)
    dt = torch.float64 if dtype == "f64" else torch.float32
    if dt == torch.float32:  # compare on FP32-representable inputs
        s.psi[:] = s.phi[:] = s.psi.astype(np.float32)
        s.c[:] = (s.c - p.cinf).astype(np.float32).astype(np.float64) + p.cinf
    ctx = lib.Context(p)
    cur, nxt = upload(p, s, dt, with_phi=True), lib.FieldSet(p, dt, with_phi=True)
    mass = torch.zeros(1, dtype=torch.float64, device="cuda")
    itip = torch.zeros(1, dtype=torch.int32, device="cuda")
    ctx.step(cur, nxt, 7, i_offset_history=2, l_offset_Vp=0.37, mass_out=mass, itip_out=itip)
    ctx.device_status()
    o = pyoracle.step(p, d, s, 7, 2, 0.37)
    g = download(p, nxt)
    tol_psi, tol_c = (1e-13, 1e-13) if dt == torch.float64 else (5e-6, 5e-8)
    assert maxabs(g.psi, o.psi) <= tol_psi and maxabs(g.phi, o.phi) <= tol_psi and maxabs(g.c, o.c) <= tol_c
    m = pyoracle.mass(p, o.c)
    assert abs(mass.item() - m) <= (1e-13 if dt == torch.float64 else 1e-8) * m
    if kind != "front" or dt == torch.float64:
        assert itip.item() == pyoracle.itip(p, o.psi)


@pytest.mark.parametrize("nx,ny", [(64, 22), (258, 32), (2048, 372), (2048, 1132)])
def test_tfc_tile_forms_match_the_oracle(nx, ny):
    """Coarse-grid temperature: 8 rows, or 16 from three waves; the polynomials
    of K + C0 and of the driving-force groups against the Gibbs functions."""
    import ctypes as C
    p = configs.small(nx, ny, i_tip_target=nx // 2, tfc=1, G=1e7, V=0.5)
    p.length_sample_um = 8.0
    p.Tcold = p.T_ref - p.GG * p.dx * p.S * p.W0 * (p.i_tip_target + 60)
    d = pyoracle.derive(p)
    L = pyoracle.lib()
    T = np.zeros(d.NxT_all * d.NyT_all)
    L.ro_initial_temperature(C.byref(p), C.byref(d), pyoracle._p(T))
    T += 0.5 * np.sin(np.arange(T.size) * 0.37)
    Tf = np.zeros((ny, nx))
    ile = d.i_left_end_initial
    L.ro_interpolate_temperature(C.byref(p), C.byref(d), pyoracle._p(T), pyoracle._p(Tf), ile)
    s = state(p, "front", nx + ny)
    ctx = lib.Context(p)
    cur, nxt = upload(p, s), lib.FieldSet(p, torch.float64)
    ctx.step(cur, nxt, 0, T_coarse=torch.from_numpy(T).cuda(), i_left_end=ile, i_left_end_T=ile)
    ctx.device_status()
    o = pyoracle.step(p, d, s, 0, T_fine=Tf)
    g = download(p, nxt)
    assert maxabs(g.psi, o.psi) <= 1e-13 and maxabs(g.c, o.c) <= 1e-13


@pytest.mark.parametrize("periodic", [1, 0])
@pytest.mark.parametrize("off", [None, -3, 0, 5])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("nx,shift", [(129, 0), (67, 0), (128, 1)])
def test_unaligned_rows_shifts_and_ghosts(nx, shift, dtype, off, periodic):
    """Odd row lengths, and aligned ones in buffers that start one element off
    (every row unaligned): with and without a fused pull-back, both boundary
    kinds, every ghost cell compared."""
    dt = torch.float64 if dtype == "f64" else torch.float32
    p = configs.small(nx, 37, i_tip_target=nx // 2, G=5e6, V=0.5, noise_amplitude=0.02, seed=9, periodic_j=periodic)
    d = pyoracle.derive(p)
    s = state(p, "front", nx)
    if dt == torch.float32:
        s.psi[:] = s.phi[:] = s.psi.astype(np.float32)
        s.c[:] = (s.c - p.cinf).astype(np.float32).astype(np.float64) + p.cinf
    ctx = lib.Context(p)
    cur, nxt = upload(p, s, dt), lib.FieldSet(p, dt, with_phi=True)
    for fs in (cur, nxt):
        for k in ("psi", "c", "phi"):
            t = getattr(fs, k)
            if t is not None and shift:
                buf = torch.empty(t.numel() + shift, dtype=dt, device="cuda")
                v = buf[shift:].view(t.shape)
                v.copy_(t)
                setattr(fs, k, v)
    ctx.step(cur, nxt, 3, i_offset_history=1, l_offset_Vp=0.2, pull_back=off)
    ctx.device_status()
    so = s if off is None else pyoracle.pull_back(p, s, off)
    o = pyoracle.step(p, d, so, 3, 1, 0.2)
    g = download(p, nxt)
    tol_psi, tol_c = (1e-13, 1e-13) if dt == torch.float64 else (5e-6, 5e-8)
    assert maxabs(g.psi, o.psi) <= tol_psi and maxabs(g.phi, o.phi) <= tol_psi and maxabs(g.c, o.c) <= tol_c


@pytest.mark.parametrize("nx", [129, 2047])
def test_unaligned_rows_with_a_network_set_stay_exact(nx):
    """Rows that are not 16-byte aligned take the exact evaluation whether or not
    a network is set, and audit nothing."""
    from rapidsolid import surrogate
    p = configs.small(nx, 40, i_tip_target=nx // 2, G=5e6, V=0.5)
    s = state(p, "front", 5)
    ctx = lib.Context(p)
    cur, a, b = upload(p, s, torch.float32), lib.FieldSet(p, torch.float32), lib.FieldSet(p, torch.float32)
    ctx.step(cur, a, 0)
    box = surrogate.fitted_box()
    box.y_scale[0] = box.y_scale[1] = 100.0
    ctx.set_surrogate(torch.from_numpy(surrogate.init_weights(1)).cuda(), box)
    ctx.step(cur, b, 0)
    assert torch.equal(a.psi, b.psi) and torch.equal(a.c, b.c)
    assert ctx.surrogate_audit()[2:] == (0, 0)
