"""Unpadded 16 and 32 px windows by how many there are: the warp-per-window kernel
while an SM holds all its windows at once, the lockstep kernel above."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _images(kind, n, rng):
    if kind == "noise":
        A = rng.random((n, n))
        return A, np.roll(A, (2, -1), (0, 1)) + 0.1 * rng.random((n, n))
    A = rng.integers(0, 2, (n, n)).astype(float)  # ties all over the planes
    A[20:50, 30:70] = 0.5
    B = np.roll(A, (1, 2), (0, 1))
    A[5, 5], B[n - 6, 7] = np.nan, np.inf
    return A, B


@pytest.mark.parametrize("kind", ["noise", "steps"])
@pytest.mark.parametrize("n_peaks", [2, 4, 5, 8])
@pytest.mark.parametrize("w,per_sm", [(16, 24), (32, 64)])
def test_same_results_in_any_number(hb, ws, w, per_sm, n_peaks, kind):
    """Windows give the same bits among few and among more than per_sm an SM, with
    and without an image mask."""
    import torch
    from hammerhead_b200 import hooks

    many = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + 37
    rng = np.random.default_rng(w + n_peaks)
    A, B = _images(kind, 150, rng)
    d = hooks.DeviceSession(ws)
    d.stage_pair(A.astype(np.float32), B.astype(np.float32))
    mask = rng.random(A.shape) < 0.05
    mask[:40, :50] = True
    p = hb.PIVParameters(window_size=w, overlap=w - 3, apodization="gauss", n_peaks=n_peaks, subpixel_method="gauss9")
    jobs = hb.pass_grid(A.shape, p)[3]
    for use in (None, mask):
        d.stage_mask(use)
        few = d.process_windows(p, jobs, want_locs=True)[:2]
        all_ = d.process_windows(p, np.resize(jobs, (many, 4)), want_locs=True)[:2]
        for a, b in zip(few, all_):
            np.testing.assert_array_equal(a, b[: len(jobs)])
            np.testing.assert_array_equal(a[: many % len(jobs)], b[many // len(jobs) * len(jobs):])
    d.stage_mask(None)


@pytest.mark.parametrize("w,n_peaks", [(16, 3), (32, 8)])
def test_time_of_few_windows(hb, ws, w, n_peaks):
    """100 windows: the default takes no longer than the best other CTA shape."""
    from hammerhead_b200 import _lib

    n = 11 * w // 2
    A, B = (np.asfortranarray(x, np.float32) for x in
            hb.synthetic.particle_pair((n, n), hb.synthetic.uniform_flow(1.3, -0.6), seed=1))
    L = _lib.lib()
    with hb.piv_workspace() as own:
        _lib.check(L.hh_stage_pair(own.ctx, _lib.fptr(A), _lib.fptr(B), n, n), own.ctx)
        d = hb.PIVParameters(window_size=w, overlap=w // 2, apodization="gauss", n_peaks=n_peaks).to_desc()
        ms, best = (ctypes.c_float * 5)(), ctypes.c_int32()
        least = [1e9] * 5
        for _ in range(5):
            _lib.check(L.hh_autotune_correlation(own.ctx, ctypes.byref(d), 5, ms, ctypes.byref(best)), own.ctx)
            least = [min(a, b) for a, b in zip(least, ms)]
    assert least[0] <= 1.2 * min(least[1:4]), least
