"""Set-up of geometries with more offset classes than the compact layout's table
holds: refused where the compact layout is asked for, the records layout and its
forces, bit for bit, where the choice is left open; a lattice set up afterwards on
the same context takes the compact layout."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("state", [False, True])
@pytest.mark.parametrize("dims", [(12, 9), (40, 41), (200, 190), (6, 5, 4), (10, 10, 9), (40, 41, 9)])
def test_more_classes_than_the_table(dims, state):
    from pd_gpu1_gb300._lib import PDError
    from pd_gpu1_gb300.engine import Engine, derive_params

    dim, dx = len(dims), 1e-3
    p = derive_params(dim, 2 if state else 1, 2, 8.7e-8, 1, dx, 1.0, dx, 0.01, 0.01, 0.01, 191e9, 0.25, 8000.0, 0.01)
    p.N = p.N_int = int(np.prod(dims))
    p.MN = 40 if dim == 2 else 160
    rng = np.random.default_rng(2)
    lattice = [g.ravel(order="F") * dx for g in np.meshgrid(*[np.arange(n) for n in dims], indexing="ij")]
    moved = [a + 0.04 * dx * rng.uniform(-1, 1, p.N) for a in lattice]
    names = ("UX", "UY", "UZ")[:dim]

    def setup(eng, coords):
        eng.set_coords(*coords)
        eng.find_neighbor_gpu()
        eng.initial_weight() if state else eng.surface_correct_gpu()
        eng.initial_state()
        eng.prepare()

    with Engine(p) as eng:
        eng.set_force_layout("compact")
        with pytest.raises(PDError, match="UNSUPPORTED"):
            setup(eng, moved)
        out = []
        for layout in ("records", "auto"):
            eng.set_force_layout(layout)
            setup(eng, moved)
            assert eng.force_layout() == "records"
            for f, a in zip(names, moved):
                eng.set(f, 1e-4 * a)
            eng.force()
            out.append([eng.get("F" + f[1]) for f in names])
        for a, b in zip(*out):
            np.testing.assert_array_equal(a, b)
        assert np.abs(out[0][0]).max() > 0.0
        setup(eng, lattice)
        assert eng.force_layout() == "compact"
