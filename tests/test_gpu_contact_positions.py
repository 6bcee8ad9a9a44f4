"""Forces after an explicit run whose last step is in contact with the impactor:
contact moves u of the touched nodes after the positions x + u of that step
were formed.  The run is a single step, so that its nodes are in contact in the
last one, twice on one context (captured, then replayed), each time further in;
the evaluation after it has to be the one after setting the same u anew, and
the context a fresh one given that state, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = ("UX", "UY", "UZ")


def _forces(eng, state):
    eng.state_force_gpu() if state else eng.bond_force_gpu()
    return {f: eng.get(f) for f in ("FX", "FY", "FZ") + (("THETA", "E") if state else ())}


@pytest.mark.parametrize("layout", ["compact", "records"])
@pytest.mark.parametrize("state", [False, True])
def test_forces_after_contact(state, layout):
    from pd_gpu1_gb300 import presets
    from pd_gpu1_gb300._abi import PD_MODEL_BOND, PD_MODEL_STATE
    from pd_gpu1_gb300.engine import Engine

    p, setup, meta = presets.build_kalthoff_winkler(scale=0.3, model=PD_MODEL_STATE if state else PD_MODEL_BOND)
    cyl = meta["cylinder"]
    with Engine(p) as eng, Engine(p) as fresh:
        for e in (eng, fresh):
            e.set_force_layout(layout)
            setup(e)
        assert eng.force_layout() == layout
        for depth in (0.2, 0.5):
            before = eng.get("UY")
            cyl.disp[1] = -depth * p.dx
            eng.cylinder_init(cyl)
            eng.run_explicit(1)
            u, fail = [eng.get(f) for f in U], eng.get("FAIL")
            # a step at 32 m/s moves a node by 0.003 dx; contact by more
            assert (np.abs(u[1] - before) > 0.05 * p.dx).sum() > 10
            got = _forces(eng, state)
            r = eng.residual()
            eng.set("FAIL", fail)
            for e in (eng, fresh):
                e.set("FAIL", fail)
                for f, v in zip(U, u):
                    e.set(f, v)
                want = _forces(e, state)
                for f in want:  # (a broken bond keeps an older extension)
                    sel = fail == 1 if f == "E" else slice(None)
                    np.testing.assert_array_equal(got[f][sel], want[f][sel], err_msg=f"{f} at {depth}")
                assert e.residual() == r
            eng.set("FAIL", fail)
            for f in ("VX", "VY", "VZ"):
                eng.set(f, np.zeros(p.N))
