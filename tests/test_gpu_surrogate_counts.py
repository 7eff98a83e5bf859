"""What rs_surrogate_audit reports does not depend on the tile height that a
step takes: the counters stand for tiles of 16 rows by 128 columns, whose rows 0
and 17 and halo columns are read, and counted, by two tiles.  A numpy count of
those tiles' network cells, and the same run inside a batched ensemble on its
16-row tiles."""
import numpy as np
import pytest

from rapidsolid import configs, lib, surrogate

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def count(psi, ny, nx):
    """Network cells of every 16 x 128 tile's box: not melt, and not in a block
    of 16 columns of solid whose 3 x 3 neighbourhood in the box is solid too."""
    n = 0
    one = np.zeros((ny + 34, nx + 300), bool)  # solid, melt of the zero-filled array, origin at (1, 4)
    melt = np.zeros_like(one)
    one[1:1 + ny, 4:4 + nx] = psi == 1.0
    melt[1:1 + ny, 4:4 + nx] = psi == -1.0
    for y0 in range(1, ny - 1, 16):
        for x0 in range(0, nx, 128):
            o = one[y0:y0 + 18, x0 + 3:x0 + 3 + 130]  # box rows, columns x0-1 .. x0+128
            m = melt[y0:y0 + 18, x0 + 3:x0 + 3 + 130].copy()
            beyond = np.arange(x0 - 1, x0 + 129) >= nx
            o = o & ~beyond
            m |= beyond
            for rr in range(18):
                if y0 - 1 + rr > ny - 1:
                    break
                a, b = max(rr - 1, 0), min(rr + 1, 17)
                col = o[a:b + 1].all(axis=0)  # solid over the rows
                if x0 == 0:
                    col[0] = True
                s3 = col[:-2] & col[1:-1] & col[2:]
                row = o[rr, 1:-1]
                if not (row.all() or row.reshape(8, 16).all(axis=1).any()):
                    s3[:] = False
                n += int((~m[rr, 1:-1] & ~s3).sum())
                for h, nb, real in ((0, 1, x0 > 0), (129, 128, x0 + 128 < nx)):
                    used = not (o[a:b + 1, h].all() and o[a:b + 1, nb].all())
                    n += int(real and not m[rr, h] and used)
    return n


# 4-row tiles below 1110 tiles of 16 rows, then 8; last tiles of 16 rows, and of 1 to 12
@pytest.mark.parametrize("nx,ny", [(388, 200), (260, 66), (512, 58), (132, 19), (640, 36), (2048, 1122), (2052, 1134)])
def test_every_network_cell_counts_as_often_as_16_row_tiles_read_it(nx, ny):
    p = configs.small(nx, ny, i_tip_target=nx // 2, G=5e6, V=0.5)
    ctx = lib.Context(p)
    a, b = lib.FieldSet(p, torch.float32), lib.FieldSet(p, torch.float32)
    j, i = np.arange(ny)[:, None], np.arange(nx)[None, :]
    front = 0.55 * nx + 0.05 * nx * np.sin(2 * np.pi * 3 * j / (ny - 2))
    psi = np.clip((front - i) / 20.0, -1.0, 1.0).astype(np.float32)
    a.psi.copy_(torch.from_numpy(psi))
    a.c.copy_(torch.from_numpy(np.where(psi == -1.0, 0.0, 1e-3).astype(np.float32)))
    w, box, _ = surrogate.train(p, n_samples=1 << 12, epochs=1, batch=1024, seed=3)
    box.T_lo, box.T_hi = 100.0, 101.0  # every cell is out of the box
    ctx.set_surrogate(w, box)
    ctx.step(a, b, 5)
    ctx.device_status()
    assert ctx.surrogate_audit()[2] == count(psi, ny, nx)


@pytest.mark.parametrize("nx,ny", [(388, 200), (260, 66), (516, 58)])
def test_a_run_alone_reports_what_it_reports_in_an_ensemble(nx, ny):
    p = configs._ti10nb(configs.default_params(), nx, ny, 5e6, 0.5, T0=configs.T_SOLIDUS_TI10NB)
    p.i_tip_target, p.noise_amplitude, p.seed = nx // 2, 0.01, 11
    w, box, _ = surrogate.train(p, n_samples=1 << 14, epochs=2, batch=1024, seed=3)
    steps = 40

    def sets(ctx):
        a, b = lib.FieldSet(p, torch.float32), lib.FieldSet(p, torch.float32)
        ctx.initial_planar(a, configs.C_LIQUID_TI10NB, configs.C_SOLID_AT_TLIQ, 7)
        return a, b

    ens = lib.Ensemble([p])
    a, b = sets(ens.ctx[0])
    ens.ctx[0].set_surrogate(w, box)
    ens.bind(0, a, b)
    ens.set_path(0)  # per-step launches, 16-row tiles
    ens.steps(steps)
    torch.cuda.synchronize()
    want = ens.ctx[0].surrogate_audit()
    ctx = lib.Context(p)
    ctx.set_surrogate(w, box)
    a, b = sets(ctx)
    hist, l, itip = 0, 0.0, torch.zeros(1, dtype=torch.int32, device="cuda")
    for n in range(steps):
        pb = None
        if n % ctx.d.step_pull_back == 0:
            ctx.itip(a, itip)
            pb = int(itip.item()) - p.i_tip_target
            hist += pb
        ctx.step(a, b, n, i_offset_history=hist, l_offset_Vp=l, pull_back=pb)
        l += p.Vp * ctx.d.dt * ctx.d.tau0 / (p.S * p.W0)
        a, b = b, a
    got = ctx.surrogate_audit()
    assert want[3] > 0
    assert tuple(got) == tuple(want)
    ens.close()


# most columns solid: last tile rows of 4, 8 and 16 rows that hold a whole tile of solid
@pytest.mark.parametrize("nx,ny", [(516, 58), (388, 200), (640, 66), (2048, 1122)])
def test_solid_tiles_report_the_cells_of_row_ny_minus_1(nx, ny):
    p = configs._ti10nb(configs.default_params(), nx, ny, 5e6, 0.5, T0=configs.T_SOLIDUS_TI10NB)
    p.i_tip_target, p.noise_amplitude, p.seed = nx // 2, 0.01, 11
    w, box, _ = surrogate.train(p, n_samples=1 << 12, epochs=1, batch=1024, seed=3)
    box.c_hi = 0.5 * (box.c_lo + box.c_hi)  # part of the cells are out of the box
    front = int(0.9 * nx)

    def step(ctx):
        a, b = lib.FieldSet(p, torch.float32), lib.FieldSet(p, torch.float32)
        ctx.initial_planar(a, configs.C_LIQUID_TI10NB, configs.C_SOLID_AT_TLIQ, 7)
        a.psi[:, : front - 20] = 1.0
        ctx.set_surrogate(w, box)
        return a, b

    ens = lib.Ensemble([p])
    ea, eb = step(ens.ctx[0])
    ens.bind(0, ea, eb)
    ens.set_path(0)  # per-step launches, 16-row tiles
    ens.steps(1)
    torch.cuda.synchronize()
    want = ens.ctx[0].surrogate_audit()
    ctx = lib.Context(p)
    a, b = step(ctx)
    tip = torch.zeros(1, dtype=torch.int32, device="cuda")
    ctx.itip(a, tip)
    pb = int(tip.item()) - p.i_tip_target
    ctx.step(a, b, 0, i_offset_history=pb, l_offset_Vp=0.0, pull_back=pb)
    assert tuple(ctx.surrogate_audit()) == tuple(want)
    assert torch.equal(b.psi, eb.psi)
    ens.close()
