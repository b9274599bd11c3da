"""General-shape windows whose planes go through L2, by how many there are: up to
one window per SM takes a round of its own, and a third round costs half as
much again as two (device time of the correlation, from the profile)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window,padding", [((77, 209), False), ((128, 128), True), ((130, 72), True)])
def test_time_of_one_and_three_rounds(hb, ws, window, padding):
    import torch
    from hammerhead_b200 import _lib, hooks

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    A, B = np.random.default_rng(1).random((2, 500, 500)).astype(np.float32)
    p = hb.PIVParameters(window_size=window, overlap=tuple(w // 2 for w in window), padding=padding, apodization="gauss")
    L, prof = _lib.lib(), (_lib.hh_kernel_profile * 5)()
    d = hooks.DeviceSession(ws)
    d.stage_pair(A, B)
    jobs = hb.pass_grid(A.shape, p)[3]
    jobs = np.concatenate([jobs] * (3 * sms // len(jobs) + 1))
    L.hh_set_profiling(ws.ctx, 1)
    try:
        def device_ms(n):
            best = 1e9
            for _ in range(6):
                _lib.check(L.hh_profile_read(ws.ctx, prof, 1), ws.ctx)
                d.process_windows(p, jobs[:n])
                _lib.check(L.hh_profile_read(ws.ctx, prof, 1), ws.ctx)
                best = min(best, prof[0].ms)
            return best

        one, two, three = device_ms(sms), device_ms(2 * sms - 6), device_ms(3 * sms - 4)
    finally:
        L.hh_set_profiling(ws.ctx, 0)
    assert one <= 0.62 * two and three <= 1.7 * two, (one, two, three)


@pytest.mark.parametrize("window,padding", [((128, 128), True), ((70, 110), True)])
def test_same_results_in_any_number(hb, ws, window, padding):
    """A window's peaks do not depend on how many are analysed with it."""
    from hammerhead_b200 import hooks

    A, B = np.random.default_rng(2).random((2, 420, 440)).astype(np.float32)
    p = hb.PIVParameters(window_size=window, overlap=tuple(w // 2 for w in window), padding=padding, apodization="gauss")
    d = hooks.DeviceSession(ws)
    d.stage_pair(A, B)
    jobs = hb.pass_grid(A.shape, p)[3]
    few = d.process_windows(p, jobs, want_locs=True)[:2]
    many = d.process_windows(p, np.concatenate([jobs] * (300 // len(jobs) + 1)), want_locs=True)[:2]
    for a, b in zip(few, many):
        np.testing.assert_array_equal(a, b[: len(jobs)])


def test_time_of_a_prime_length(hb, ws):
    """Rows of 41 points against rows of 40: the 41 outputs of each are dealt over
    the CTA's threads, so the direct sums cost a few times the transform of 40
    points, not sixteen times."""
    from hammerhead_b200 import _lib, hooks

    A, B = np.random.default_rng(4).random((2, 300, 300)).astype(np.float32)
    L, prof = _lib.lib(), (_lib.hh_kernel_profile * 5)()
    d = hooks.DeviceSession(ws)
    d.stage_pair(A, B)
    L.hh_set_profiling(ws.ctx, 1)
    ms = []
    try:
        for cols in (40, 41):
            p = hb.PIVParameters(window_size=(14, cols), overlap=(7, 20))
            jobs, best = hb.pass_grid(A.shape, p)[3][:100], 1e9
            for _ in range(6):
                _lib.check(L.hh_profile_read(ws.ctx, prof, 1), ws.ctx)
                d.process_windows(p, jobs)
                _lib.check(L.hh_profile_read(ws.ctx, prof, 1), ws.ctx)
                best = min(best, prof[0].ms)
            ms.append(best)
    finally:
        L.hh_set_profiling(ws.ctx, 0)
    assert ms[1] <= 6 * ms[0], ms
