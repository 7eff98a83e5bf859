"""The z march of the 3D kernels through fields that change between pure melt
and fronts several times within a chunk, in whole planes and in parts of them.

One step against the FP64 oracle, and every z chunk length bit for bit the
same.  Tolerances: FP64 1e-13 (as the one-step oracle test); FP32 64 ulp of 1,
2^-24 each: every term of an update is below 1 in size (dt lambda = 0.45,
dt (2 / dx^2) 3 = 0.36) and some 50 roundings add up.  Ti-Nb in FP32: the
roundings of mu are 16 ulp of its span, and reach c by the six faces of a cell,
cf (S + S') each; those of phi are 64 ulp of 1 + the largest update."""
import numpy as np
import pytest
import torch

import pyoracle
from rapidsolid import configs, lib, surrogate
from test_gpu_peri3d import params, run_gpu, to_gpu, to_host

pytestmark = pytest.mark.gpu

TOL = {torch.float64: 1e-13, torch.float32: 64 * 2.0**-24}


def fields(p, seed, off, base, span=0.01):
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
    d = (base - off + span * (r.random(shape) - 0.5)).astype(np.float32)
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
    same_for_every_chunk(lambda chunk: params(*shape, G_T=-2e-4, z_T=12.0, z_chunk=chunk), f, dtype)


def same_for_every_chunk(make, f, dtype):
    base = run_gpu(make(0), f, 3, dtype)
    for chunk in (1, 2, 5, 64):
        for x, y in zip(run_gpu(make(chunk), f, 3, dtype), base):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("well", [0.0, 2.0])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("shape", [(4, 4, 4), (64, 16, 33), (68, 17, 40), (132, 31, 70), (36, 15, 5)])
def test_tinb_changes_between_melt_and_fronts(shape, dtype, well):
    """c within 0.0125 of c_ref = 0.9: both sides of the melt polynomial's range."""

    def make(chunk):
        p = configs.tinb_3d(nx=shape[0], ny=shape[1], nz=shape[2], z_front=12.0)
        p.z_chunk, p.a1 = chunk, well
        p.Da = 0.1 * well
        return p

    p = make(0)
    f = fields(p, sum(shape), p.c_ref, p.c_ref, 0.025)
    out, ref = run_gpu(p, f, 1, dtype), pyoracle.run3(p, f, 1)
    if dtype == torch.float64:
        tol_phi = tol_c = 1e-13 * (1.0 + max(np.abs(a - b).max() for a, b in zip(ref, f)))
    else:
        ulp = 2.0**-24
        cf = 0.5 * p.dt * p.alpha * p.dx_inv**2
        s_max = max(1.0, 0.25 * p.AA**2 / (p.AA - 1.0)) * 0.1 * 0.9 * 1.2 + 0.1 * well * 0.1
        tol_phi = 64 * ulp * (1.0 + max(np.abs(ref[i] - f[i]).max() for i in (0, 1)))
        tol_c = 64 * ulp + 6 * cf * 2 * s_max * 16 * ulp * np.ptp(pyoracle.mu3(p, *f))
    assert max(np.abs(out[i] - ref[i]).max() for i in (0, 1)) <= tol_phi
    assert np.abs(out[2] - ref[2]).max() <= tol_c
    same_for_every_chunk(make, f, dtype)


def test_surrogate_counters_do_not_depend_on_the_chosen_chunk():
    """z_chunk = 0 picks a chunk by the volume; the audit's counters stay those
    of a march in chunks of 32 planes, and so do the fields."""
    p = configs.tinb_3d(nx=68, ny=31, nz=70, z_front=12.0)
    p2 = configs.scale()
    p2.cinf = p.c_ref
    w, box, _ = surrogate.train(p2, box=surrogate.fitted_box(), n_samples=1 << 14, epochs=1, batch=4096, seed=3,
                                g_input=True)
    f = fields(p, 7, p.c_ref, p.c_ref, 0.1)
    out = []
    for chunk in (0, 32):
        p.z_chunk = chunk
        ctx = lib.Context3(p)
        ctx.set_surrogate(w, box)
        a, b = to_gpu(p, f, torch.float32), lib.FieldSet3(p, torch.float32)
        for k in range(3):
            ctx.step(a, b, k)
            a, b = b, a
        torch.cuda.synchronize()
        ctx.device_status()
        out.append((to_host(a, p), ctx.surrogate_audit()))
        ctx.close()
    assert out[0][1] == out[1][1] and out[0][1][3] > 0
    for x, y in zip(out[0][0], out[1][0]):
        assert np.array_equal(x, y)
