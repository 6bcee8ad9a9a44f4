"""The forms of the 2-D bond kernel for small problems work on every slot row of
a warp whether its bonds are used or not.  On plates 40 nodes wide, where two of
five slot rows hold padding, with a tenth of the bonds broken and the two halves
of the plate apart by 50 spacings (broken bonds far from their classes): the
one-warp kernel's results bit for bit, at a size of each form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _start(eng):
    eng.initial_state()
    x, y, dx = eng.get("X"), eng.get("Y"), eng.p.dx
    rowptr, nl = eng.csr()
    row = np.repeat(np.arange(eng.p.N), np.diff(rowptr))
    cut = (x[row] < 0) != (x[nl] < 0)
    # the same random tenth from both ends
    lo, hi = np.minimum(row, nl).astype(np.int64), np.maximum(row, nl).astype(np.int64)
    cut |= (lo * 7919 + hi * 104729) % 10 == 0
    eng.set("FAIL", np.where(cut, 0, 1).astype(np.int32))
    rng = np.random.default_rng(3)
    eng.set("UX", np.where(x > 0, 50 * dx, 0.0) + 1e-3 * (0.3 * x + 0.05 * dx * rng.standard_normal(eng.p.N)))
    eng.set("UY", 1e-3 * (y + 0.05 * dx * rng.standard_normal(eng.p.N)))


# 113, 500, 875, 1125 and 1875 slices: 8, 4 and 2 warps a slice, two slots a lane
@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("ny", [90, 400, 700, 900, 1500])
def test_unused_slots_change_nothing(ny, mode):
    from pd_gpu1_gb300.engine import Engine, derive_params

    nx, dx = 40, 5e-4
    p = derive_params(2, 1, mode, 1.0 if mode == 1 else 5e-8, 1, dx, 0.0, dx, nx * dx, ny * dx, 0.0, 192e9, 1.0 / 3.0,
                      8000.0, 1.1e-3)
    p.nx, p.ny, p.N_int, p.N = nx, ny, nx * ny, nx * ny + 6 * nx
    out = []
    with Engine(p) as eng:
        eng.coord_plate_crack()
        eng.find_neighbor_gpu()
        eng.surface_correct_gpu()
        for waves in (1, 2):
            eng.set_launch(256, 0, waves, 1)
            _start(eng)
            if mode == 1:
                eng.run_adr(0, 6, 0.0)
            else:
                eng.run_explicit(6, load=1.0, dmg_every=6)
            eng.bond_force_gpu()
            out.append({f: eng.get(f) for f in ("UX", "UY", "VX", "VY", "FX", "FY", "FAIL")})
    assert np.isfinite(out[0]["FX"]).all() and (out[0]["FAIL"] == 0).mean() > 0.1
    for f in out[0]:
        np.testing.assert_array_equal(out[0][f], out[1][f], err_msg=f)
