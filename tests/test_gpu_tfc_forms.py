"""Coarse-grid temperature on the tile kernels, against the oracle: rows that are
not 16-byte aligned (odd lengths, and aligned ones in buffers one element off) and
aligned ones, both precisions, tiles of 8 and 16 rows, fused pull-backs, a front
and deep solid (the whole-tile form).  Tolerances as with the frozen temperature
(test_gpu_tile_forms.py): the groups are the same functions of the cell's
temperature, rounded alike."""
import ctypes as C

import numpy as np
import pytest

import pyoracle
from helpers import maxabs
from rapidsolid import configs, lib
from test_gpu_step import download, upload
from test_gpu_tile_forms import state

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def run(nx, ny, dtype, kind, off, shift):
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
    s = state(p, kind, nx + ny)
    dt = torch.float64 if dtype == "f64" else torch.float32
    if dt == torch.float32:
        s.psi[:] = s.phi[:] = s.psi.astype(np.float32)
        s.c[:] = (s.c - p.cinf).astype(np.float32).astype(np.float64) + p.cinf
    ctx = lib.Context(p)
    cur, nxt = upload(p, s, dt), lib.FieldSet(p, dt, with_phi=True)
    if shift:
        for fs in (cur, nxt):
            for k in ("psi", "c", "phi"):
                t = getattr(fs, k)
                if t is not None:
                    buf = torch.empty(t.numel() + shift, dtype=dt, device="cuda")
                    v = buf[shift:].view(t.shape)
                    v.copy_(t)
                    setattr(fs, k, v)
    mass = torch.zeros(1, dtype=torch.float64, device="cuda")
    ctx.step(cur, nxt, 0, T_coarse=torch.from_numpy(T).cuda(), i_left_end=ile, i_left_end_T=ile, pull_back=off,
             mass_out=mass)
    ctx.device_status()
    o = pyoracle.step(p, d, s if off is None else pyoracle.pull_back(p, s, off), 0, T_fine=Tf)
    g = download(p, nxt)
    tol_psi, tol_c = (1e-13, 1e-13) if dt == torch.float64 else (5e-6, 5e-8)
    assert maxabs(g.psi, o.psi) <= tol_psi and maxabs(g.phi, o.phi) <= tol_psi and maxabs(g.c, o.c) <= tol_c
    m = pyoracle.mass(p, o.c)
    assert abs(mass.item() - m) <= (1e-13 if dt == torch.float64 else 1e-8) * m


@pytest.mark.parametrize("off", [None, -3, 5])
@pytest.mark.parametrize("kind", ["front", "solid"])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("nx,ny,shift", [(65, 22, 0), (129, 32, 0), (257, 42, 0), (128, 22, 1), (256, 42, 1),
                                         (256, 42, 0), (2049, 372, 0)])
def test_coarse_temperature_tiles_match_the_oracle(nx, ny, shift, dtype, kind, off):
    run(nx, ny, dtype, kind, off, shift)


# 16-row tiles in FP64 (three waves)
@pytest.mark.parametrize("off", [None, 5])
@pytest.mark.parametrize("nx,shift", [(2049, 0), (2050, 1)])
def test_coarse_temperature_16_row_tiles_on_unaligned_rows(nx, shift, off):
    run(nx, 1132, "f64", "front", off, shift)


# the line between 8 and 16 rows in FP64 (1073 tiles of 16 x 64 on a B200): 1072, 1088, 1088 tiles
@pytest.mark.parametrize("off", [None, 5])
@pytest.mark.parametrize("nx,ny", [(1024, 1072), (1024, 1082), (1023, 1082)])
def test_coarse_temperature_at_the_line_between_the_tile_heights(nx, ny, off):
    run(nx, ny, "f64", "front", off, 0)
