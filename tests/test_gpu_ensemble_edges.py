"""The persistent walk over runs that are mostly far melt, with a last tile column
that reaches beyond the array: a CTA fills those columns of its input tile by
ordinary stores, leaves the tile by the far-melt form, and the next tile's load
lands in the same shared memory.  Every path must equal the per-step launches
bit for bit."""
import numpy as np
import pytest

from rapidsolid import configs, lib

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# last tile columns of 4, 64 and 124 cells; more tiles than CTAs fit on the device in every tile shape
RUNS = [(1924, 1030), (1216, 1540), (1020, 2050), (772, 1282)]
STEPS = 24


def run(path):
    ps, ens = [], None
    for k, (nx, ny) in enumerate(RUNS):
        p = configs._ti10nb(configs.default_params(), nx, ny, 5e6, 0.5, T0=configs.T_SOLIDUS_TI10NB)
        p.i_tip_target, p.noise_amplitude, p.seed = 16, 0.01, 40 + k
        ps.append(p)
    ens = lib.Ensemble(ps)
    for r, p in enumerate(ps):
        a, b = lib.FieldSet(p, torch.float32), lib.FieldSet(p, torch.float32)
        ens.ctx[r].initial_planar(a, configs.C_LIQUID_TI10NB, configs.C_SOLID_AT_TLIQ, 7)
        # solute noise inside the far-melt bound, so that stale columns would be seen
        g = torch.Generator(device="cuda")
        g.manual_seed(r)
        a.c += 5e-5 * (2 * torch.rand(a.c.shape, device="cuda", generator=g) - 1) * (a.psi == -1.0)
        ens.bind(r, a, b)
    ens.set_path(path)
    ens.steps(STEPS)
    torch.cuda.synchronize()
    ens.ctx[0].device_status()
    out = [(f.psi.cpu().numpy(), f.c.cpu().numpy()) for f in (ens.state(r)[3] for r in range(len(ps)))]
    ens.close()
    return out


def test_walk_with_far_melt_edge_tiles_equals_per_step_launches():
    want = run(0)
    melt = [float((psi[:, psi.shape[1] // 2:] == -1.0).mean()) for psi, _ in want]
    assert min(melt) > 0.99
    for path in (3, 5, 10, 15, 17):
        for r, ((psi, c), (psi0, c0)) in enumerate(zip(run(path), want)):
            assert np.array_equal(psi, psi0) and np.array_equal(c, c0), (path, r)
