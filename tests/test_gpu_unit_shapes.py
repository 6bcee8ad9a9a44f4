"""The state-based passes and the 3-D bond kernel of the compact layout take
another number of slot phases at each problem size (8, 4, 2 or 1).  At sizes
around each limit: forces, dilatation and intact flags against the 48- and
32-byte records, whose bond vectors are rounded as the reference rounds them,
with small displacements and with ones that turn the specimen by 0.2 rad (bond
vectors outside their classes' binades); and an explicit run in one call
against the same steps in two.

A bond vector differs between the layouts by the roundings of its ends'
positions and of the differences, four units of 2^-53 of the largest position P
in all; forces go with the extensions, which are of the random displacements'
size sigma, so they may differ by 4 2^-53 P / sigma, next to the 2e-13 of the
pair arithmetic."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the limits are 2, 6 and 12 slices per SM in 2-D (152 SMs): 304, 912, 1824
PLATES = [60, 95, 96, 167, 168, 238, 239]
# and 4, 10, 24 and 32 in 3-D: 608, 1520, 3648, 4864
SLABS = [0.3, 0.4, 0.6, 0.8, 1.0]


def _compare(p, setup, fields, force, sigma, turn, broken):
    from pd_gpu1_gb300.engine import Engine

    rng = np.random.default_rng(3)
    u = sigma * rng.standard_normal((len(fields), p.N))
    out = {}
    with Engine(p) as eng:
        for layout in ("compact", "records"):
            eng.set_force_layout(layout)
            setup(eng)
            assert eng.force_layout() == layout
            x, y = eng.get("X"), eng.get("Y")
            c, s = np.cos(turn) - 1.0, np.sin(turn)
            for f, v, r in zip(fields, u, (c * x - s * y, s * x + c * y, 0.0)):
                eng.set(f, v + r)
            force(eng)
            first = [eng.get("F" + f[1]) for f in fields]
            force(eng)  # on the bonds that the first pass left
            out[layout] = first, [eng.get("F" + f[1]) for f in fields], eng.get("THETA"), eng.get("FAIL")
        pmax = max(np.abs(x).max(), np.abs(y).max()) * 1.5
        tol = 4 * 2.0**-53 * pmax / sigma + 2e-13
        n = p.N_int
        got, want = out["compact"], out["records"]
        for a, b in zip(got[0] + got[1], want[0] + want[1]):
            assert np.linalg.norm(a[:n] - b[:n]) <= tol * np.linalg.norm(b[:n])
        assert np.linalg.norm(got[2] - want[2]) <= tol * np.linalg.norm(want[2]) + 1e-300
        np.testing.assert_array_equal(got[3], want[3])
        if broken:
            assert (got[3] == 0).sum() > 1000


def _run(p, setup, fields, load, steps, motion=None):
    from pd_gpu1_gb300.engine import Engine

    out = []
    with Engine(p) as eng:
        for parts in ([steps], [steps // 2, steps - steps // 2]):
            setup(eng)
            if motion is not None:
                eng.cylinder_init(motion)
            for k in parts:
                eng.run_explicit(k, load=load)
            out.append([eng.get(f) for f in fields] + [eng.get("FAIL")])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("turn", [0.0, 0.2])
@pytest.mark.parametrize("nx", PLATES)
def test_state_plate(nx, turn):
    from pd_gpu1_gb300 import presets

    p, setup, _ = presets.build_crack_grow(scale=nx / 500.0)
    assert p.nx == nx
    _compare(p, setup, ("UX", "UY"), lambda e: e.state_force_gpu(), 2.5e-6, turn, True)


@pytest.mark.parametrize("nx", PLATES)
def test_state_plate_steps(nx):
    from pd_gpu1_gb300 import presets

    p, setup, meta = presets.build_crack_grow(scale=nx / 500.0)
    _run(p, setup, ("UX", "UY", "VX", "VY", "FX", "FY", "THETA"), meta["load"], 7)


@pytest.mark.parametrize("turn", [0.0, 0.2])
@pytest.mark.parametrize("state", [False, True])
@pytest.mark.parametrize("scale", SLABS)
def test_slab(scale, state, turn):
    from pd_gpu1_gb300 import presets
    from pd_gpu1_gb300._abi import PD_MODEL_BOND, PD_MODEL_STATE

    p, setup, _ = presets.build_kalthoff_winkler(scale=scale, model=PD_MODEL_STATE if state else PD_MODEL_BOND)
    _compare(p, setup, ("UX", "UY", "UZ"), lambda e: e.state_force_gpu() if state else e.bond_force_gpu(), 1e-5, turn,
             True)


@pytest.mark.parametrize("state", [False, True])
@pytest.mark.parametrize("scale", SLABS)
def test_slab_steps(scale, state):
    from pd_gpu1_gb300 import presets
    from pd_gpu1_gb300._abi import PD_MODEL_BOND, PD_MODEL_STATE

    p, setup, meta = presets.build_kalthoff_winkler(scale=scale, model=PD_MODEL_STATE if state else PD_MODEL_BOND)
    cyl = meta["cylinder"]
    cyl.disp[1] = -0.3 * p.dx  # in contact from the first step
    _run(p, setup, ("UX", "UY", "UZ", "VY", "FX", "FY", "FZ"), 0.0, 7, cyl)
