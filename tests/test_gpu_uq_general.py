"""Uncertainty statistics of the general form at the smallest windows, with
fewer pixels than threads, and on both sides of the size whose buffers still
fit in shared memory (44 x 64 does, 48 x 60 does not)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [(4, 6), (6, 4), (9, 31), (44, 64), (48, 60)])
def test_general_uncertainty_edges(ws, orc, hb, w):
    from hammerhead_b200 import hooks, synthetic

    A, B = synthetic.particle_pair((160, 192), synthetic.uniform_flow(1.4, -0.8), seed=5)
    p = hb.PIVParameters(window_size=w, overlap=(w[0] // 2, w[1] // 2), padding=True, apodization="gauss",
                         uncertainty=True)
    sess = hooks.DeviceSession(ws)
    sess.stage_pair(A, B)
    jobs = hb.pass_grid(A.shape, p)[3]
    jobs = np.concatenate([jobs[:3], jobs[-3:]])
    _, _, uq = sess.process_windows(p, jobs, want_uq=True)
    for q, (_, _, rs, cs) in enumerate(jobs):
        win = np.s_[rs - 1:rs - 1 + w[0], cs - 1:cs - 1 + w[1]]
        s = orc.uq_stats(A[win].astype(np.float64), B[win].astype(np.float64), "gauss", dtype=np.float64)
        # per-pixel Float32 values of O(1), sums in double: 2e-5 of the
        # component's largest sum covers n roundings of 2^-24 each
        for comp in (0, 1):
            c = slice(44 * comp, 44 * comp + 44)
            np.testing.assert_allclose(uq[q, c], s[c], rtol=0, atol=2e-5 * np.abs(s[c]).max())
