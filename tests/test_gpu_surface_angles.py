"""The surface coefficient of 3-D bonds whose coordinate differences lie on the
1e-10 at which the angle's branches change: half of the nodes of a lattice
column shifted by it, so that bonds have differences of 1e-10, just below and
zero beside lattice ones.  Within 1e-13 of the oracle, the bar of the goldens,
from several set-ups (the remembered angles are shared by every thread)."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axes", [(0,), (1,), (0, 1)])
def test_differences_at_the_branch_limit(axes):
    from pd_gpu1_gb300.engine import Engine, derive_params

    n, dx = 15, 1e-3
    p = derive_params(3, 1, 2, 8.7e-8, 1, dx, 1.0, dx, n * dx, n * dx, n * dx, 191e9, 0.25, 8000.0, 0.01)
    p.N = p.N_int = n**3
    p.MN = 128
    k, j, i = np.meshgrid(*[np.arange(n) - n // 2] * 3, indexing="ij")
    c = [a.ravel() * dx for a in (i, j, k)]
    for a in axes:  # the column at coordinate 0, where 1e-10 is a difference exactly
        at = c[a] == 0.0
        layer = k.ravel() % 3
        c[a][at & (layer == 1)] = 1e-10
        c[a][at & (layer == 2)] = np.nextafter(1e-10, 0.0)
        assert {0.0, 1e-10} <= set(c[a])
    m = orc.Model(p, *c)
    m.find_neighbor()
    m.surface_correct()
    want = m.rows(m.scr)
    with Engine(p) as eng:
        for _ in range(3):
            eng.set_coords(*c)
            eng.find_neighbor_gpu()
            eng.surface_correct_gpu()
            np.testing.assert_allclose(eng.get("SCR"), want, rtol=1e-13, atol=0)


def _lattice(dims, dx, jitter, seed=5):
    rng = np.random.default_rng(seed)
    grids = np.meshgrid(*[np.arange(n) - n // 2 for n in dims], indexing="ij")
    return [g.ravel(order="F") * dx + jitter * dx * rng.uniform(-1, 1, g.size) for g in grids]


# up to 72 rows an SM a warp per row, a thread beyond: 10,944 at 152 SMs
@pytest.mark.parametrize("jitter", [0.0, 0.05])
@pytest.mark.parametrize("dims", [(5, 3), (33, 31), (104, 105), (105, 105), (4, 3, 2), (11, 12, 9), (34, 35, 9), (35, 35, 9)])
def test_warp_and_thread_per_row(dims, jitter):
    """Within 1e-13 of the oracle on both sides of the limit, on and off the
    lattice, and the same from both ends of a bond, bit for bit."""
    from pd_gpu1_gb300.engine import Engine, derive_params

    dim, dx = len(dims), 1e-3
    c = _lattice(dims, dx, jitter)
    p = derive_params(dim, 1, 2, 8.7e-8, 1, dx, 1.0, dx, 0.01, 0.01, 0.01, 191e9, 0.25, 8000.0, 0.01)
    p.N = p.N_int = len(c[0])
    p.MN = 40 if dim == 2 else 160
    m = orc.Model(p, *c)
    m.find_neighbor()
    m.surface_correct()
    with Engine(p) as eng:
        eng.set_coords(*c)
        eng.find_neighbor_gpu()
        eng.surface_correct_gpu()
        scr = eng.get("SCR")
        rowptr, nl = eng.csr()
    np.testing.assert_allclose(scr, m.rows(m.scr), rtol=1e-13, atol=0)
    row = np.repeat(np.arange(p.N), np.diff(rowptr)).astype(np.int64)
    there, back = np.lexsort((nl, row)), np.lexsort((row, nl))
    np.testing.assert_array_equal(scr[there], scr[back])
