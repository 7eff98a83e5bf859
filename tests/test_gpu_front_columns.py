"""The front at the border of two tile columns of a tall FP32 grid, where a step
takes 16-row tiles: the fields of the lower tiles that it takes with the front
elsewhere, bit for bit, and the same counters."""
import numpy as np
import pytest

from rapidsolid import configs, lib, surrogate

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# tile columns 2, 3 and 4 of 128; ny - 2 beyond 14, 16, 18, 20 and 24 rows per SM of a B200
@pytest.mark.parametrize("network", [False, True])
@pytest.mark.parametrize("nx,ny", [(192, 2300), (260, 2390), (260, 2702), (448, 3000), (388, 3600)])
def test_fields_do_not_depend_on_where_the_front_is_said_to_be(nx, ny, network):
    out = []
    for tip in (64, 114, 134, 10):  # beside the offset, made up for below, i_tip_target orders the tiles and chooses their height
        p = configs._ti10nb(configs.default_params(), nx, ny, 5e6, 0.5, T0=configs.T_SOLIDUS_TI10NB)
        p.i_tip_target, p.noise_amplitude, p.seed = tip, 0.01, 5
        ctx = lib.Context(p)
        a, b = lib.FieldSet(p, torch.float32), lib.FieldSet(p, torch.float32)
        if not out:
            p.i_tip_target = 128
            lib.Context(p).initial_planar(a, configs.C_LIQUID_TI10NB, configs.C_SOLID_AT_TLIQ, 7)
            start = a.psi.clone(), a.c.clone()
        a.psi.copy_(start[0])
        a.c.copy_(start[1])
        if network:
            w, box, _ = surrogate.train(p, n_samples=1 << 12, epochs=1, batch=1024, seed=3)
            ctx.set_surrogate(w, box)
        mass = torch.zeros(12, dtype=torch.float64, device="cuda")
        for n in range(12):
            ctx.step(a, b, n, i_offset_history=tip - 64, l_offset_Vp=0.01 * n, pull_back=1 if n == 5 else None,
                     mass_out=mass[n:n + 1] if n % 2 else None)
            a, b = b, a
        ctx.device_status()
        out.append((a.psi.cpu(), a.c.cpu(), ctx.surrogate_audit() if network else None, mass.cpu().numpy()))
    for x in out[1:]:
        assert torch.equal(x[0], out[0][0]) and torch.equal(x[1], out[0][1])
        assert x[2] == out[0][2]
        assert np.allclose(x[3], out[0][3], rtol=1e-13)  # FP64 sums of the same cells in another order
