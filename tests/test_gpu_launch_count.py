"""hh_launch_count against the kernels that ran (the CUDA activity trace): single
pairs and ensembles with and without a mask, predictor smoothing and a
convergence test. Rectangular windows, whose correlation is one kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ensemble", [False, True])
@pytest.mark.parametrize("smoothing", [True, False])
@pytest.mark.parametrize("masked", [False, True])
def test_counts_the_kernels_that_ran(hb, ws, masked, smoothing, ensemble):
    import torch
    from hammerhead_b200 import _lib
    from torch.profiler import ProfilerActivity, profile

    A, B = hb.synthetic.particle_pair((240, 220), hb.synthetic.uniform_flow(1.3, -0.6), seed=1)
    mask = None
    if masked:
        mask = np.zeros(A.shape, bool)
        mask[:90, :70] = True
    more = {} if ensemble else dict(max_iterations=3, convergence_tol=1e-9)
    passes = [hb.PIVParameters(window_size=(48, 32), overlap=(24, 16), **more) for _ in range(2)]

    def run():
        if ensemble:
            hb.run_piv_ensemble([(A, B)] * 2, passes, workspace=ws, mask=mask, predictor_smoothing=smoothing)
        else:
            hb.run_piv(A, B, passes, workspace=ws, mask=mask, predictor_smoothing=smoothing)

    run()
    torch.zeros(1, device="cuda")
    count = _lib.lib().hh_launch_count
    before = count(ws.ctx)
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        run()
    booked = count(ws.ctx) - before
    ran = [e.name for e in p.events() if "hh::" in e.name]
    if not ran:
        pytest.skip("no activity trace here")
    assert booked == len(ran), sorted(ran)
