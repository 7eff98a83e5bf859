"""The z march of the 3D kernels through fields that change between pure melt
and fronts several times within a chunk, in whole planes and in parts of them.

One step against the FP64 oracle, and every z chunk length bit for bit the
same.  Tolerances: FP64 1e-13 (as the one-step oracle test); FP32 64 ulp of 1,
2^-24 each: every term of an update is below 1 in size (dt lambda = 0.45,
dt (2 / dx^2) 3 = 0.36) and some 50 roundings add up."""
import numpy as np
import pytest
import torch

import pyoracle
from rapidsolid import lib
from test_gpu_peri3d import params, run_gpu

pytestmark = pytest.mark.gpu

TOL = {torch.float64: 1e-13, torch.float32: 64 * 2.0**-24}


def fields(p, seed, off, base):
    """Melt with slabs, single planes, single cells and a corner of mixed phase;
    the values are FP32 (c - off), ghost layers as images."""
    r = np.random.default_rng(seed)
    shape = (p.nz, p.ny, p.nx)
    a = np.ones(shape, np.float32)
    b = np.zeros(shape, np.float32)
    mixed = np.zeros(shape, bool)
    for z in range(p.nz):
        kind = r.integers(0, 6)
        if kind == 0:
            mixed[z] = True
        elif kind == 1:
            mixed[z, r.integers(0, p.ny), r.integers(0, p.nx)] = True
        elif kind == 2:
            mixed[z, : p.ny // 2, p.nx // 3 :] = True
    a[mixed] = r.random(mixed.sum(), np.float32)
    b[mixed] = (1.0 - a[mixed]) * r.random(mixed.sum(), np.float32)
    d = (base - off + 0.01 * (r.random(shape) - 0.5)).astype(np.float32)
    out = [a.astype(np.float64), b.astype(np.float64), d.astype(np.float64) + off]
    for f in out:  # periodic x, y; no-flux z
        f[:, :, 0], f[:, :, -1] = f[:, :, -2], f[:, :, 1].copy()
        f[:, 0], f[:, -1] = f[:, -2], f[:, 1].copy()
        f[0], f[-1] = f[1], f[-2]
    return out


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("shape", [(4, 4, 4), (64, 16, 33), (68, 17, 40), (132, 31, 70), (36, 15, 5)])
def test_changes_between_melt_and_fronts(shape, dtype):
    p = params(*shape, G_T=-2e-4, z_T=12.0)
    off = lib.c_offset3(p)
    f = fields(p, sum(shape), off, off)
    out = run_gpu(p, f, 1, dtype)
    ref = pyoracle.run3(p, f, 1)
    for x, y in zip(out, ref):
        assert np.abs(x - y).max() <= TOL[dtype]
    for chunk in (1, 2, 5, 64):
        q = params(*shape, G_T=-2e-4, z_T=12.0, z_chunk=chunk)
        for x, y in zip(run_gpu(q, f, 3, dtype), run_gpu(p, f, 3, dtype)):
            assert np.array_equal(x, y)
