"""The tip's row scan and the grid reductions at the sizes where their passes
change over: more rows than one read of the scan (2048) and one more or less,
rows shorter and longer than one turn of the column walk (512 cells), odd row
lengths, fronts that raise the tip in every row, in none, or with ties.  The
scan's comparisons are the oracle's, so i, j and status agree exactly; x, y and
R differ by the rounding of the same fits (the tolerances of the fixture
test)."""
import ctypes as C

import numpy as np
import pytest

import pyoracle
from rapidsolid import _abi, configs, lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def front(nx, ny, shape, seed):
    rng = np.random.default_rng(seed)
    j = np.arange(ny)
    mid, amp = 0.5 * nx, 0.35 * nx
    i0 = {"rise": mid + amp * (j / ny - 0.5), "fall": mid - amp * (j / ny - 0.5), "flat": np.full(ny, mid),
          "cells": mid + amp * np.sin(j / 17.0), "noise": mid + amp * (2 * rng.random(ny) - 1),
          "melt": np.full(ny, -50.0), "solid": np.full(ny, 2.0 * nx)}[shape]
    return -np.tanh((np.arange(nx)[None, :] - i0[:, None]) * 0.8 / np.sqrt(2.0))


@pytest.mark.parametrize("shape", ["rise", "fall", "flat", "cells", "noise", "melt", "solid"])
@pytest.mark.parametrize("nx,ny", [(24, 33), (129, 2047), (513, 2048), (96, 2049), (1100, 70), (64, 4100)])
def test_scan_and_reductions_match_the_oracle(nx, ny, shape):
    p = configs.small(nx, ny, i_tip_target=nx // 2)
    d = pyoracle.derive(p)
    psi = front(nx, ny, shape, nx + ny)
    ctx = lib.Context(p)
    fs = lib.FieldSet(p, torch.float64)
    fs.psi.copy_(torch.from_numpy(psi))
    fs.c.copy_(torch.from_numpy(0.9 + 0.01 * psi))
    tip = torch.zeros(C.sizeof(_abi.Tip), dtype=torch.uint8, device="cuda")
    itip = torch.zeros(1, dtype=torch.int32, device="cuda")
    mass = torch.zeros(1, dtype=torch.float64, device="cuda")
    ctx.itip(fs, itip)
    ctx.precise_tip(fs, tip)
    ctx.mass(fs, mass)
    t, o = lib.tip_from_bytes(tip.cpu().numpy().tobytes()), pyoracle.precise_tip(p, d, psi)
    assert itip.item() == pyoracle.itip(p, psi)
    assert (t.i, t.j, t.status) == (o.i, o.j, o.status)
    for k, tol in (("x", 1e-12), ("y", 1e-12), ("R", 1e-9)):
        a, b = getattr(t, k), getattr(o, k)
        assert (a == b) or (np.isnan(a) and np.isnan(b)) or abs(a - b) <= tol * max(1.0, abs(b)), k
    m = pyoracle.mass(p, 0.9 + 0.01 * psi)
    assert abs(mass.item() - m) <= 1e-13 * m


def test_output_turn_in_a_captured_graph():
    p = configs.small(256, 96, i_tip_target=40)
    ctx = lib.Context(p)
    a, b = lib.FieldSet(p, torch.float64), lib.FieldSet(p, torch.float64)
    ctx.initial_planar(a, configs.C_LIQUID_TI10NB, configs.C_SOLID_AT_TLIQ, 3)
    tip = torch.zeros(C.sizeof(_abi.Tip), dtype=torch.uint8, device="cuda")
    itip = torch.zeros(1, dtype=torch.int32, device="cuda")
    mass = torch.zeros(1, dtype=torch.float64, device="cuda")

    def turn():
        tip.zero_()
        ctx.step(a, b, 0, mass_out=mass)
        ctx.itip(b, itip)
        ctx.precise_tip(b, tip)
        ctx.mass(b, mass)
        b.psi.add_(0.0)

    turn()
    torch.cuda.synchronize()
    want = [x.clone() for x in (tip, itip, mass, b.psi, b.c)]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        turn()
    for x in (tip, itip, mass, b.psi, b.c):
        x.fill_(1)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    for x, w in zip((tip, itip, mass, b.psi, b.c), want):
        assert torch.equal(x, w)
