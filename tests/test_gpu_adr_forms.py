"""A single specimen's ADR steps take two warps a slice up to 8 slices an SM and
one beyond.  On both sides of the limit: displacements, damping coefficient and
residual of the two-wave shape of the one-warp kernel, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 1213, 1220 slices of 32 rows; the limit is 1216 at 152 SMs
@pytest.mark.parametrize("nx,ny", [(197, 197), (198, 197)])
def test_adr_on_both_sides_of_eight_slices_an_sm(nx, ny):
    from pd_gpu1_gb300.engine import Engine, derive_params

    dx = 5e-4
    p = derive_params(2, 1, 1, 1.0, 1, dx, 0.0, dx, nx * dx, ny * dx, 0.0, 192e9, 1.0 / 3.0, 8000.0, 1.1e-3)
    p.nx, p.ny, p.N_int, p.N = nx, ny, nx * ny, nx * ny + 6 * nx
    out = []
    with Engine(p) as eng:
        eng.coord_plate_crack()
        eng.find_neighbor_gpu()
        eng.surface_correct_gpu()
        x, y = eng.get("X"), eng.get("Y")
        for waves in (1, 2):
            eng.set_launch(256, 0, waves, 1)
            eng.initial_state()
            eng.set_crack_2d(nx * dx / 3.0, 0.0, 0.0, 0.3)
            rng = np.random.default_rng(7)
            eng.set("UX", 1e-3 * (0.3 * x + 0.05 * dx * rng.standard_normal(p.N)))
            eng.set("UY", 1e-3 * (y + 0.05 * dx * rng.standard_normal(p.N)))
            it, r = eng.adr_solve(0, 12, 6, 0.0)
            out.append({f: eng.get(f) for f in ("UX", "UY", "VHX", "VHY", "FX", "FY", "FAIL")})
            out[-1].update(residual=np.array([r]), cn=np.array([eng.adr_cn()]))
    assert out[0]["residual"][0] > 0.0 and (out[0]["FAIL"] == 0).sum() > 100
    for f in out[0]:
        np.testing.assert_array_equal(out[0][f], out[1][f], err_msg=f)
