"""The smoothing passes of the warm-start prediction against numpy: each free
node's mean over itself and its intact neighbours, prescribed rows counting as
zero, on plates whose row count is no multiple of 32, with a pre-crack, on both
force layouts.  The correction is taken from the two candidates' difference, so
it carries a rounding of the increment: the bar is eight units of it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,layout,passes", [(41, 37, "compact", 1), (41, 37, "records", 2), (9, 5, "compact", 3),
                                                 (130, 71, "compact", 5)])
def test_smoothing_is_the_family_mean(nx, ny, layout, passes):
    import torch

    from pd_gpu1_gb300._lib import check, lib
    from pd_gpu1_gb300.engine import Engine, derive_params
    from pd_gpu1_gb300.warm import Net, init_params

    dx = 1e-4
    p = derive_params(2, 1, 1, 1.0, 1, dx, 0.0, dx, nx * dx, ny * dx, 0.0, 192e9, 1.0 / 3.0, 8000.0, 8e-3)
    p.nx, p.ny, p.N_int, p.N = nx, ny, nx * ny, nx * ny + 6 * nx
    q = init_params(2)
    q[-258:] = np.random.default_rng(4).standard_normal(258).astype(np.float32)
    net = Net(1024, q)
    with Engine(p) as eng:
        eng.set_force_layout(layout)
        eng.coord_plate_crack()
        eng.find_neighbor_gpu()
        eng.surface_correct_gpu()
        eng.initial_state()
        eng.set_crack_2d(0.6 * nx * dx, 0.0, 0.0, 0.2)
        x, y = eng.get("X"), eng.get("Y")
        eng.set("UX", 1e-4 * x)
        eng.set("UY", 2e-4 * y)
        n = p.N_int
        du = torch.zeros(4 * n, dtype=torch.float64, device="cuda")
        out = []
        for k in (0, passes):
            check(lib().pd_warm_predict(eng.ctx, net.h, 1e-5, 5e-7, k, du.data_ptr(), None), eng.ctx, "predict")
            out.append(du.cpu().numpy().copy())
        rowptr, nl = eng.csr()
        alive = eng.get("FAIL") == 1
    net.close()
    np.testing.assert_array_equal(out[0][2 * n:], out[1][2 * n:])
    bar = 8 * np.finfo(float).eps * np.abs(out[0]).max()
    moved = 0.0
    for a in range(2):
        skip = out[0][(2 + a) * n:(3 + a) * n]
        c0 = c = out[0][a * n:(a + 1) * n] - skip
        for _ in range(passes):
            new = np.empty(n)
            for i in range(n):
                nb = nl[rowptr[i]:rowptr[i + 1]][alive[rowptr[i]:rowptr[i + 1]]]
                new[i] = (c[i] + c[nb[nb < n]].sum()) / (1 + nb.size)
            c = new
        got = out[1][a * n:(a + 1) * n] - skip
        assert np.abs(got - c).max() <= bar, a
        moved = max(moved, np.abs(c - c0).max())
    assert moved > 100 * bar
