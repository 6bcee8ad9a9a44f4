"""The slot phases of the 3-D kernels on both sides of each of their limits, the
larger ones included: 4, 30 and 48 slices an SM in the dilatation pass, 4 and 48
in the state-based force pass, 10 and 32 in the bond kernel (152 SMs: 608, 1520,
4560, 4864 and 7296 slices).  The comparisons and bars of test_gpu_unit_shapes:
forces, dilatation and intact flags against the records layout, and a run in one
call against the same steps in two."""
import pytest

from test_gpu_unit_shapes import _compare, _run

pytestmark = pytest.mark.gpu

STATE = {0.32: 585, 0.33: 632, 0.89: 4506, 0.895: 4581, 1.13: 7247, 1.135: 7342}
BOND = {0.51: 1492, 0.52: 1535, 0.92: 4787, 0.925: 4891}


def _slab(scale, state, slices):
    from pd_gpu1_gb300 import presets
    from pd_gpu1_gb300._abi import PD_MODEL_BOND, PD_MODEL_STATE

    out = presets.build_kalthoff_winkler(scale=scale, model=PD_MODEL_STATE if state else PD_MODEL_BOND)
    assert (out[0].N + 31) // 32 == slices
    return out


CASES = [(s, True, n) for s, n in STATE.items()] + [(s, False, n) for s, n in BOND.items()]


@pytest.mark.parametrize("turn", [0.0, 0.2])
@pytest.mark.parametrize("scale,state,slices", CASES)
def test_slab(scale, state, slices, turn):
    p, setup, _ = _slab(scale, state, slices)
    _compare(p, setup, ("UX", "UY", "UZ"), lambda e: e.state_force_gpu() if state else e.bond_force_gpu(), 1e-5, turn,
             True)


@pytest.mark.parametrize("scale,state,slices", CASES)
def test_slab_steps(scale, state, slices):
    p, setup, meta = _slab(scale, state, slices)
    cyl = meta["cylinder"]
    cyl.disp[1] = -0.3 * p.dx  # in contact from the first step
    _run(p, setup, ("UX", "UY", "UZ", "VY", "FX", "FY", "FZ"), 0.0, 7, cyl)
