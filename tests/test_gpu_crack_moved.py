"""Pre-crack flags where the caller has written new coordinates into the context's
own memory after the family was built: bonds then reach further than its
horizon, and every one has to be looked at.  Against the oracle, whose family is
the unstretched plate's as well."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("theta", [0.0, 0.3, np.pi / 2, 1.5, -0.8])
def test_flags_after_coordinates_were_written(theta):
    import torch

    from pd_gpu1_gb300.engine import Engine, derive_params

    nx, ny, dx = 61, 43, 5e-4
    p = derive_params(2, 1, 2, 1e-7, 1, dx, 0.0, dx, 0.01, 0.01, 0.0, 192e9, 1.0 / 3.0, 8000.0, 0.04472)
    p.N = p.N_int = nx * ny
    p.MN = 32
    i, j = np.meshgrid(np.arange(nx), np.arange(ny))
    x, y = ((-nx / 2.0 + 0.5 + i) * dx).ravel(), ((-ny / 2.0 + 0.5 + j) * dx).ravel()
    crack = (2.0 * nx * dx, 1e-4, -2e-4, theta)
    m = orc.Model(p, x.copy(), y.copy())
    m.find_neighbor()
    near = orc.Model(p, x.copy(), y.copy())
    near.find_neighbor()
    near.set_crack_2d(*crack)
    m.x[:], m.y[:] = 3.0 * x, 3.0 * y
    m.set_crack_2d(*crack)
    want = m.rows(m.fail)
    assert (want == 0).sum() > 0 and (want != near.rows(near.fail)).any()
    with Engine(p) as eng:
        eng.set_coords(x, y)
        eng.find_neighbor_gpu()
        eng.initial_state()
        eng.device_view("X").copy_(torch.from_numpy(3.0 * x))
        eng.device_view("Y").copy_(torch.from_numpy(3.0 * y))
        eng.set_crack_2d(*crack)
        np.testing.assert_array_equal(eng.get("FAIL"), want)


# up to 72 rows an SM a warp per row, a thread beyond: 10,944 at 152 SMs
@pytest.mark.parametrize("theta", [0.0, 0.3, np.pi / 2, 1.5, -0.8])
@pytest.mark.parametrize("nx,ny", [(7, 5), (61, 43), (104, 105), (105, 105), (171, 150)])
def test_flags_on_both_sides_of_the_limit(nx, ny, theta):
    from pd_gpu1_gb300.engine import Engine, derive_params

    dx = 5e-4
    p = derive_params(2, 1, 2, 1e-7, 1, dx, 0.0, dx, 0.01, 0.01, 0.0, 192e9, 1.0 / 3.0, 8000.0, 0.04472)
    p.N = p.N_int = nx * ny
    p.MN = 32
    i, j = np.meshgrid(np.arange(nx), np.arange(ny))
    x, y = ((-nx / 2.0 + 0.5 + i) * dx).ravel(), ((-ny / 2.0 + 0.5 + j) * dx).ravel()
    crack = (0.7 * ny * dx, 1e-4, -2e-4, theta)
    m = orc.Model(p, x, y)
    m.find_neighbor()
    m.set_crack_2d(*crack)
    want = m.rows(m.fail)
    assert (want == 0).sum() > 0
    with Engine(p) as eng:
        eng.set_coords(x, y)
        eng.find_neighbor_gpu()
        eng.initial_state()
        eng.set_crack_2d(*crack)
        np.testing.assert_array_equal(eng.get("FAIL"), want)
