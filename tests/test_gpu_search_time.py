"""Device time of enlarged search areas against windows of the area's size, 2500 of
each: the same transforms, a second mean, and more pixels a thread than its
registers hold (36 at 48 and 96 px), which must not spill."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,window,method,most", [(96, 88, "cross", 2.15), (48, 40, "phase", 1.9)])
def test_search_area_against_window(hb, ws, size, window, method, most):
    from hammerhead_b200 import _lib, hooks

    A, B = hb.synthetic.particle_pair((700, 700), hb.synthetic.uniform_flow(1.3, -0.6), seed=1)
    L, prof = _lib.lib(), (_lib.hh_kernel_profile * 5)()
    d = hooks.DeviceSession(ws)
    d.stage_pair(A, B)
    L.hh_set_profiling(ws.ctx, 1)
    try:
        def device_ms(w):
            p = hb.PIVParameters(window_size=w, search_area_size=size, overlap=w // 2, apodization="gauss",
                                 correlation_method=method)
            jobs, best = np.resize(hb.pass_grid(A.shape, p)[3], (2500, 4)), 1e9
            for _ in range(8):
                _lib.check(L.hh_profile_read(ws.ctx, prof, 1), ws.ctx)
                d.process_windows(p, jobs)
                _lib.check(L.hh_profile_read(ws.ctx, prof, 1), ws.ctx)
                best = min(best, prof[0].ms)
            return best

        search, plain = device_ms(window), device_ms(size)
    finally:
        L.hh_set_profiling(ws.ctx, 0)
    assert search <= most * plain, (search, plain)
