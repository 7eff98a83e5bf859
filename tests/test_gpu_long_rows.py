"""Unaligned rows longer than the FP64 tile kernels' grid (65535 tile columns):
the register kernel takes the step."""
import numpy as np
import pytest

import pyoracle
from helpers import fix_ghosts, maxabs
from rapidsolid import configs, lib
from test_gpu_step import download, upload

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_a_row_of_more_than_65535_tiles():
    nx, ny = 64 * 65535 + 65, 8
    p = configs.small(nx, ny, i_tip_target=nx - 300, G=1e3, V=0.05)
    d = pyoracle.derive(p)
    s = pyoracle.initial_planar(p, configs.C_LIQUID_TI10NB, configs.C_SOLID_AT_TLIQ, 3)
    x = (np.arange(nx) - p.i_tip_target) * p.dx / np.sqrt(2.0)
    s.psi[:] = s.phi[:] = -np.tanh(x)[None, :]
    s.c[:] = p.cinf + 1e-3 * np.sin(np.arange(nx) * 0.01)[None, :] * (1 + s.psi) / 2
    fix_ghosts(p, s)
    ctx = lib.Context(p)
    cur, nxt = upload(p, s), lib.FieldSet(p, torch.float64)
    ctx.step(cur, nxt, 3)
    ctx.device_status()
    o = pyoracle.step(p, d, s, 3)
    g = download(p, nxt)
    assert maxabs(g.psi, o.psi) <= 1e-13 and maxabs(g.c, o.c) <= 1e-13
