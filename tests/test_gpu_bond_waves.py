"""An explicit step or a force evaluation of 28 to 32 slices an SM takes the form
of the one-warp kernel with fewer registers, which forms a bond's components one
after the other: the bits of the other form, on both sides of both limits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 4255, 4266, 4864 and 4876 slices; the limits are 4256 and 4864 at 152 SMs
@pytest.mark.parametrize("nx,ny", [(364, 374), (365, 374), (394, 395), (395, 395)])
def test_forms_agree(nx, ny):
    from pd_gpu1_gb300.engine import Engine, derive_params

    dx = 5e-4
    p = derive_params(2, 1, 2, 5e-8, 1, dx, 0.0, dx, nx * dx, ny * dx, 0.0, 192e9, 1.0 / 3.0, 8000.0, 1.1e-3)
    p.nx, p.ny, p.N_int, p.N = nx, ny, nx * ny, nx * ny + 6 * nx
    out = []
    with Engine(p) as eng:
        eng.coord_plate_crack()
        eng.find_neighbor_gpu()
        eng.surface_correct_gpu()
        x, y = eng.get("X"), eng.get("Y")
        for block in (256, 512):
            eng.set_launch(block, 0, 1, 1)
            eng.initial_state()
            eng.set_crack_2d(nx * dx / 3.0, 0.0, 0.0, 0.3)
            rng = np.random.default_rng(11)
            eng.set("UX", 1e-3 * (0.3 * x + 0.05 * dx * rng.standard_normal(p.N)))
            eng.set("UY", 1e-3 * (y + 0.05 * dx * rng.standard_normal(p.N)))
            eng.run_explicit(6, load=1.0, dmg_every=6)
            eng.bond_force_gpu()
            out.append({f: eng.get(f) for f in ("UX", "UY", "VX", "VY", "FX", "FY", "FAIL", "DMG")})
    assert (out[0]["FAIL"] == 0).sum() > 100
    for f in out[0]:
        np.testing.assert_array_equal(out[0][f], out[1][f], err_msg=f)
