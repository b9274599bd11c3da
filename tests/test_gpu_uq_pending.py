"""Uncertainties of the register form, which finalizes the windows of several
iterations together: fewer windows than a warp keeps, a remainder, and several
rounds of every warp; with and without a mask. The run's sigma is the oracle's
finalize_uncertainty of the statistics the same kernel reports (logarithms in
double on both sides, one rounding to Float32: 1e-6 relative)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,size,step", [(8, 40, 3), (12, 16, 4), (16, 16, 8), (16, 72, 8), (16, 600, 3), (24, 24, 12),
                                         (24, 560, 4), (32, 40, 8), (32, 600, 5)])
@pytest.mark.parametrize("masked", [False, True])
def test_pending_windows(ws, orc, hb, w, size, step, masked):
    from hammerhead_b200 import hooks, synthetic

    A, B = synthetic.particle_pair((size, size + 7), synthetic.uniform_flow(1.4, -0.8), seed=9)
    p = hb.PIVParameters(window_size=w, overlap=w - step, padding=True, apodization="gauss", uncertainty=True,
                         uod_enable=False, replace_outliers=False)
    mask = None
    if masked:
        mask = np.zeros(A.shape, bool)
        mask[size // 2:, : size // 3] = True
        mask[0, 0] = True
    res = hb.run_piv(A, B, p, mask=mask, workspace=ws)
    _, _, _, jobs = hb.pass_grid(A.shape, p, mask)
    sess = hooks.DeviceSession(ws)
    sess.stage_pair(A, B)
    sess.stage_mask(mask)
    _, _, uq = sess.process_windows(p, jobs, want_uq=True)
    sess.stage_mask(None)
    pick = np.unique(np.concatenate([np.arange(min(len(jobs), 40)), np.arange(max(len(jobs) - 40, 0), len(jobs)),
                                     np.arange(0, len(jobs), 97)]))
    for q in pick:
        gi, gj = jobs[q, 0] - 1, jobs[q, 1] - 1
        for comp, unc in ((0, res.uncertainty_u), (1, res.uncertainty_v)):
            want = orc.finalize_uncertainty(uq[q, 44 * comp:44 * comp + 44])
            np.testing.assert_allclose(unc[gi, gj], want, rtol=1e-6, equal_nan=True)
