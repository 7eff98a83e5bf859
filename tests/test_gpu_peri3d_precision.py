"""Rounding of the FP64 3D TiAg step's solute: its error against an 80-bit
evaluation of the model stays near what rounding mu once per cell would leave."""
import numpy as np
import pytest

from rapidsolid import configs, lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

LD = np.longdouble


def at(f, o=(0, 0, 0)):
    n = f.shape
    return f[1 + o[2]:n[0] - 1 + o[2], 1 + o[1]:n[1] - 1 + o[1], 1 + o[0]:n[2] - 1 + o[0]]


def mu_exact(p, p1, p2, c):
    """mu = c - sum r_i g_i (computeMu, TiAg.cu:461-470) in 80 bits."""
    p1, p2, c = (v.astype(LD) for v in (p1, p2, c))
    p3 = 1 - p1 - p2
    g = lambda a, b, d: a * a / 4 * (15 * (1 - a) * (1 + a - (d - b) ** 2) + a * (9 * a * a - 5))  # noqa: E731
    A1, A2 = LD(p.A1), LD(p.A2)
    return c - A1 * g(p1, p2, p3) + (A1 + A2) * g(p2, p3, p1) + (A1 - A2) * g(p3, p1, p2)


def solute(p, p1, c, mu):
    """c' (TiAg.cu:543-552) from mu, in 80 bits."""
    p1, c, mu = (v.astype(LD) for v in (p1, c, mu))
    dc = LD(0)
    for o, h in (((1, 0, 0), p.dx_inv), ((0, 1, 0), p.dy_inv), ((0, 0, 1), p.dz_inv)):
        for s in (1, -1):
            q = tuple(s * v for v in o)
            dc = dc + (at(p1, q) + at(p1)) / 2 * (at(mu, q) - at(mu)) * LD(h) * LD(h)
    return at(c) + LD(p.dt) * LD(p.alpha) * dc


def test_solute_error_is_that_of_one_rounding_of_mu():
    p = configs.peritectic_3d(nx=48, ny=40, nz=48)
    rng = np.random.default_rng(2)
    z, y, x = np.meshgrid(np.arange(p.nz), np.arange(p.ny), np.arange(p.nx), indexing="ij")
    h = 0.5 * (1 + np.tanh((z - 16 - 3 * np.sin(2 * np.pi * 2 * x / (p.nx - 2))) / 2.0))
    share = 0.5 * (1 + np.tanh(3.0 * np.sin(2 * np.pi * 3 * y / (p.ny - 2) + 0.3)))
    p1, p2 = h, (1 - h) * share
    c = 0.3 * h - 0.3 * p2 + 0.5 * (1 - h - p2) + 0.002 * h * np.exp(-np.abs(z - 16) / 8.0) * rng.random(h.shape)
    for f in (p1, p2, c):  # ghost cells: x and y periodic, z held
        f[:, :, 0], f[:, :, -1] = f[:, :, -2], f[:, :, 1]
        f[:, 0], f[:, -1] = f[:, -2], f[:, 1]
        f[0], f[-1] = f[1], f[-2]
    ctx = lib.Context3(p)
    a, b = lib.FieldSet3(p, torch.float64), lib.FieldSet3(p, torch.float64)
    for t, f in ((a.phi1, p1), (a.phi2, p2), (a.c, c)):
        t.copy_(torch.from_numpy(f))
    ctx.step(a, b, 0)
    ctx.device_status()
    mu = mu_exact(p, p1, p2, c)
    want = solute(p, p1, c, mu)
    rms = lambda e: float(np.sqrt(np.mean(e.astype(LD) ** 2)))  # noqa: E731
    # one rounding of mu and one of c'; the three terms' own roundings may add 40 %
    least = rms(solute(p, p1, c, mu.astype(np.float64)).astype(np.float64) - want)
    assert rms(at(b.c.cpu().numpy()) - want) <= 1.4 * least
