"""The branches of the family build and the set-up passes at the sizes where
they change: families of rows up to 32, up to 128 and longer (the three row
writers), a box so large that the single-precision distance filter stands
aside, pre-cracks at every kind of angle, the surface coefficient off the
lattice (no operand pair repeats), and a second set-up on the same context
(its memory is the first one's)."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu


def _engine(p):
    from pd_gpu1_gb300.engine import Engine

    return Engine(p)


def _derive(n, dx, model=1, MN=0):
    from pd_gpu1_gb300.engine import derive_params

    p = derive_params(2, model, 2, 1e-7, 1, dx, 0.0, dx, 0.01, 0.01, 0.0, 192e9, 1.0 / 3.0, 8000.0, 0.04472)
    p.N = p.N_int = n
    p.MN = MN
    return p


@pytest.mark.parametrize("horizon,shift", [(3.015, 0.0), (6.0, 0.0), (8.0, 0.0), (3.015, 3e6)])
def test_family_of_a_random_cloud(horizon, shift):
    """28, 113 and 201 members in the mean, and a cloud with one node millions
    of horizons away (exact predicate throughout), against all pairs with the
    reference's predicate."""
    n, dx = 3000, 1e-3
    rng = np.random.default_rng(int(horizon * 10))
    side = np.sqrt(n) * dx
    x, y = rng.uniform(0, side, n), rng.uniform(0, side, n)
    if shift:
        x[0] = shift * dx
        x[1], y[1] = x[2] + horizon * dx, y[2]  # on the horizon, to rounding
    p = _derive(n, dx)
    p.delta = horizon * dx
    with _engine(p) as eng:
        eng.set_coords(x, y)
        eng.find_neighbor_gpu()
        rowptr, nl = eng.csr()
    for i in range(n):
        dx_, dy_ = x - x[i], y - y[i]
        want = np.flatnonzero(dx_ * dx_ + dy_ * dy_ < p.delta * p.delta)
        np.testing.assert_array_equal(nl[rowptr[i]:rowptr[i + 1]], want[want != i])


def _jittered(nx, ny, dx, jitter, seed=3):
    i, j = np.meshgrid(np.arange(nx), np.arange(ny))
    rng = np.random.default_rng(seed)
    x = ((-nx / 2.0 + 0.5 + i) * dx).ravel() + jitter * dx * rng.uniform(-1, 1, nx * ny)
    y = ((-ny / 2.0 + 0.5 + j) * dx).ravel() + jitter * dx * rng.uniform(-1, 1, nx * ny)
    return x, y


@pytest.mark.parametrize("theta,frac,lx,ly", [(0.0, 0.5, 0.0, 0.0), (0.3, 0.7, 1e-3, -2e-3), (np.pi / 2, 0.4, 2.5e-4, 0.0),
                                              (1.5, 0.9, 0.0, 1e-3), (-0.8, 3.0, 0.0, 0.0), (0.0, 0.5, 0.0, 2.5e-4)])
def test_pre_crack_flags_match_the_oracle(theta, frac, lx, ly):
    nx, ny, dx = 61, 43, 5e-4
    x, y = _jittered(nx, ny, dx, 0.0)
    p = _derive(nx * ny, dx, MN=32)
    m = orc.Model(p, x, y)
    m.find_neighbor()
    m.set_crack_2d(frac * nx * dx, lx, ly, theta)
    with _engine(p) as eng:
        eng.set_coords(x, y)
        eng.find_neighbor_gpu()
        eng.initial_state()
        eng.set_crack_2d(frac * nx * dx, lx, ly, theta)
        np.testing.assert_array_equal(eng.get("FAIL"), m.rows(m.fail))
    assert (m.rows(m.fail) == 0).sum() > 0


@pytest.mark.parametrize("nx,ny,jitter", [(40, 30, 0.0), (97, 65, 0.05)])
def test_surface_coefficient_and_rebuild(nx, ny, jitter):
    """scr within 1e-13 of the oracle (the bar of the goldens) on a lattice
    and on one where no two bonds share their angle (more operand pairs than
    the table holds), the same bits from a second set-up on the context and
    after another family in between."""
    dx = 5e-4
    x, y = _jittered(nx, ny, dx, jitter)
    p = _derive(nx * ny, dx, MN=40)
    m = orc.Model(p, x, y)
    m.find_neighbor()
    m.surface_correct()
    with _engine(p) as eng:
        def build(xs, ys):
            eng.set_coords(xs, ys)
            eng.find_neighbor_gpu()
            eng.surface_correct_gpu()
            eng.initial_state()
            eng.set("UX", 1e-4 * xs)
            eng.prepare()
            eng.bond_force_gpu()
            return [eng.get(f) for f in ("NL", "IDIST", "FAC", "SCR", "FX", "FY")]

        first = build(x, y)
        want = m.rows(m.scr)
        np.testing.assert_allclose(first[3], want, rtol=1e-13, atol=0)
        np.testing.assert_array_equal(first[1], m.rows(m.idist))
        np.testing.assert_array_equal(first[2], m.rows(m.fac))
        build(0.9 * x, 0.9 * y)
        for a, b in zip(first, build(x, y)):
            np.testing.assert_array_equal(a, b)
