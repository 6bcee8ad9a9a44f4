"""Contexts are independent: a prediction, and the set-up of a new context, do not
wait for what another stream of the process is doing (a kernel that takes some
tenths of a second here), and a prediction after a set-up on another stream that
it was ordered behind gives what it gives on one stream."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BUSY = 1_000_000_000  # clock cycles, about half a second


def _plate(stream=None):
    from pd_gpu1_gb300.engine import Engine, derive_params

    nx, ny, dx = 130, 71, 1e-4
    p = derive_params(2, 1, 1, 1.0, 1, dx, 0.0, dx, nx * dx, ny * dx, 0.0, 192e9, 1.0 / 3.0, 8000.0, 8e-3)
    p.nx, p.ny, p.N_int, p.N = nx, ny, nx * ny, nx * ny + 6 * nx
    return Engine(p, stream=stream)


def _setup(eng):
    eng.coord_plate_crack()
    eng.find_neighbor_gpu()
    eng.surface_correct_gpu()
    eng.initial_state()
    eng.prepare()


def _predictor(eng, passes):
    import torch

    from pd_gpu1_gb300._lib import check, lib
    from pd_gpu1_gb300.warm import Net, init_params

    net = Net(1024, init_params(2))
    du = torch.zeros(4 * eng.p.N_int, dtype=torch.float64, device="cuda")

    def run():
        check(lib().pd_warm_predict(eng.ctx, net.h, 1e-5, 5e-7, passes, du.data_ptr(), eng.stream), eng.ctx, "predict")
        return du

    return run


@pytest.mark.parametrize("passes", [0, 3])
def test_prediction_does_not_wait_for_another_stream(passes):
    import torch

    side = torch.cuda.Stream()
    with _plate() as eng:
        _setup(eng)
        eng.set("UX", 1e-4 * eng.get("X"))
        run = _predictor(eng, passes)
        run()
        torch.cuda.synchronize()
        done = torch.cuda.Event()
        with torch.cuda.stream(side):
            torch.cuda._sleep(BUSY)
            done.record()
        run()
        waited = done.query()
        torch.cuda.synchronize()
    assert not waited


def test_setup_of_a_new_context_does_not_wait_for_another_stream():
    import torch

    side = torch.cuda.Stream()
    with _plate() as first:
        _setup(first)  # the library's kernels loaded
    with _plate() as eng:
        torch.cuda.synchronize()
        done = torch.cuda.Event()
        with torch.cuda.stream(side):
            torch.cuda._sleep(BUSY)
            done.record()
        _setup(eng)
        eng.sync()
        waited = done.query()
        torch.cuda.synchronize()
        forces = eng.get("NN")
    assert not waited and forces.max() > 0


def test_prediction_on_another_stream_after_a_rebuild():
    """Set-up on one stream, prediction on another that waits for it: the blocks
    that the set-up gave back are not taken while its kernels read them."""
    import torch

    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with _plate(a.cuda_stream) as eng:
        _setup(eng)
        ux, uy = 1e-4 * eng.get("X"), 2e-4 * eng.get("Y")
        run = _predictor(eng, 3)

        def passes(on):
            out = []
            for _ in range(5):
                eng.stream = a.cuda_stream
                _setup(eng)
                eng.set("UX", ux)
                eng.set("UY", uy)
                b.wait_stream(a)
                eng.stream = on.cuda_stream
                out.append(run().cpu().numpy().copy())
            eng.stream = a.cuda_stream
            return out

        want = passes(a)[0]
        for got in passes(b):
            np.testing.assert_array_equal(got, want)
