"""The compact layout on a lattice with differences of 1e-23 and -1e-23 between
the coordinates of one column: an offset class of its own each, too small for a
scale as a float.  The layout takes it, and forces, dilatation and flags are the
records layout's to the bars of test_gpu_unit_shapes, unturned and turned (the
bond's component then is far from its class's)."""
import numpy as np
import pytest

from test_gpu_unit_shapes import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("turn", [0.0, 0.2])
@pytest.mark.parametrize("state", [False, True])
@pytest.mark.parametrize("n", [41, 301])
def test_component_below_the_scale(n, state, turn):
    from pd_gpu1_gb300.engine import derive_params

    dx = 1e-4
    p = derive_params(2, 2 if state else 1, 2, 1.3367e-8, 1, dx, 0.0, dx, n * dx, n * dx, 0.0, 192e9, 0.3, 7850.0,
                      0.04472)
    p.nx = p.ny = n
    p.N = p.N_int = n * n
    j, i = np.meshgrid(np.arange(n) - n // 2, np.arange(n) - n // 2, indexing="ij")
    x, y = i.ravel() * dx, j.ravel() * dx
    at = x == 0.0
    x[at & (j.ravel() % 2 == 1)] = 1e-23
    assert len(set(x[at])) == 2

    def setup(eng):
        eng.set_coords(x, y)
        eng.find_neighbor_gpu()
        if state:
            eng.initial_weight()
        else:
            eng.surface_correct_gpu()
        eng.initial_state()
        eng.prepare()

    _compare(p, setup, ("UX", "UY"), lambda e: e.state_force_gpu() if state else e.bond_force_gpu(), 2.5e-6, turn,
             False)
