"""The default launch shape of the 2-D bond kernels takes another form at each
problem size (8, 4 or 2 warps per slice, two slots side by side, one warp per
slice).  Each has to give the one-warp kernel's results bit for bit, bonds that
break, ADR's grid-wide damping and residual sums and a batch's per-specimen
ones included.  The one-warp kernel is asked for by its two-wave shape, which
at these sizes runs the same blocks as the default one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# slices (of 32 interior rows) around the limits 1, 4, 6, 12 and 16 per SM at 152 SMs
SIZES = [(37, 29), (70, 69), (71, 70), (139, 140), (140, 141), (170, 171), (171, 172), (241, 242), (278, 279), (290, 290)]


def _plate(nx, ny, mode, s0):
    from pd_gpu1_gb300.engine import Engine, derive_params

    dx = 5e-4
    p = derive_params(2, 1, mode, 1.0 if mode == 1 else 5e-8, 1, dx, 0.0, dx, nx * dx, ny * dx, 0.0, 192e9, 1.0 / 3.0,
                      8000.0, s0)
    p.nx, p.ny, p.N_int, p.N = nx, ny, nx * ny, nx * ny + 6 * nx
    eng = Engine(p)
    eng.coord_plate_crack()
    eng.find_neighbor_gpu()
    eng.surface_correct_gpu()
    return eng


def _start(eng, seed, strain):
    eng.initial_state()
    eng.set_crack_2d(eng.p.nx * eng.p.dx / 3.0, 0.0, 0.0, 0.3)
    rng = np.random.default_rng(seed)
    x, y = eng.get("X"), eng.get("Y")
    eng.set("UX", strain * (0.3 * x + 0.05 * eng.p.dx * rng.standard_normal(eng.p.N)))
    eng.set("UY", strain * (y + 0.05 * eng.p.dx * rng.standard_normal(eng.p.N)))


def _same(a, b):
    for f in a:
        np.testing.assert_array_equal(a[f], b[f], err_msg=f)


@pytest.mark.parametrize("nx,ny", SIZES)
def test_explicit_steps(nx, ny):
    out = []
    with _plate(nx, ny, 2, 1.1e-3) as eng:
        for waves in (1, 2):
            eng.set_launch(256, 0, waves, 1)
            _start(eng, 5, 1e-3)
            eng.run_explicit(6, load=1.0, dmg_every=6)
            eng.bond_force_gpu()
            out.append({f: eng.get(f) for f in ("UX", "UY", "VX", "VY", "FX", "FY", "FAIL", "DMG")})
    assert (out[0]["FAIL"] == 0).sum() > 100
    _same(*out)


@pytest.mark.parametrize("nx,ny", SIZES)
def test_adr_steps(nx, ny):
    out = []
    with _plate(nx, ny, 1, 1.1e-3) as eng:
        for waves in (1, 2):
            eng.set_launch(256, 0, waves, 1)
            _start(eng, 7, 1e-3)
            it, r = eng.adr_solve(0, 12, 6, 0.0)
            out.append({f: eng.get(f) for f in ("UX", "UY", "VHX", "VHY", "FX", "FY", "FAIL")})
            out[-1].update(residual=np.array([r]), cn=np.array([eng.adr_cn()]))
    assert out[0]["residual"][0] > 0.0 and (out[0]["FAIL"] == 0).sum() > 100
    _same(*out)


@pytest.mark.parametrize("sides", [(20, 33), (60, 47, 90), (120, 101, 80)])
def test_batch_steps(sides):
    from pd_gpu1_gb300.engine import Batch, derive_params

    base = derive_params(2, 1, 1, 1.0, 1, 5e-4, 0.0, 5e-4, 0.05, 0.05, 0.0, 192e9, 1.0 / 3.0, 8000.0, 0.04472)
    specs = [dict(nx=n, ny=n + 1, emod=(70 + 10 * k) * 1e9, critical_s=1e-3 * (1 + k), crack_len=0.2 * n * 5e-4,
                  crack_theta=0.4 * k, load_scale=1.0 + 0.1 * k) for k, n in enumerate(sides)]
    out = []
    for waves in (1, 2):
        with Batch(base, specs) as eng:
            eng.set_launch(256, 0, waves, 1)
            eng.run_adr(0, 15, 2.7e-6)
            out.append({f: eng.get(f) for f in ("UX", "UY", "FX", "FY", "FAIL")})
            out[-1]["cn"] = eng.cn()
    _same(*out)


@pytest.mark.parametrize("nx,ny", [(623, 624), (624, 624), (701, 650)])  # the limit is 80 slices per SM: 12160
def test_large_adr_sums(nx, ny):
    """From 80 slices an SM the damping sums go through memory, except in a step
    that forms the residual: one at every step against one at every sixth.  From
    rest with the boundary rows pulled apart, where the damping is positive."""
    out = []
    with _plate(nx, ny, 1, 1.1e-3) as eng:
        for check in (1, 6):
            eng.initial_state()
            y = eng.get("Y")
            eng.set("UY", np.where(np.arange(eng.p.N) >= eng.p.N_int, 1e-3 * eng.p.dx * np.sign(y), 0.0))
            it, r = eng.adr_solve(0, 12, check, 0.0)
            assert it == 12
            out.append({f: eng.get(f) for f in ("UX", "UY", "VHX", "VHY", "FX", "FY", "FAIL")})
            out[-1].update(residual=np.array([r]), cn=np.array([eng.adr_cn()]))
    assert out[0]["residual"][0] > 0.0 and out[0]["cn"][0] > 0.0
    _same(*out)


@pytest.mark.parametrize("nx,ny", [(279, 279), (331, 300), (500, 401)])  # from 16 slices per SM: 2432
def test_explicit_waves(nx, ny):
    """Explicit steps of 16 slices an SM and more run in small blocks and several
    waves: the bits of one wave of large blocks."""
    out = []
    with _plate(nx, ny, 2, 1.1e-3) as eng:
        for block in (256, 512):
            eng.set_launch(block, 0, 1, 1)
            _start(eng, 11, 1e-3)
            eng.run_explicit(6, load=1.0, dmg_every=6)
            eng.bond_force_gpu()
            out.append({f: eng.get(f) for f in ("UX", "UY", "VX", "VY", "FX", "FY", "FAIL", "DMG")})
    assert (out[0]["FAIL"] == 0).sum() > 100
    _same(*out)
