"""Validation with 3 and 4 layers of neighbours, whose medians sort local arrays,
beside 1 and 2 layers, which run in registers: batches of both against single
pairs, and the time of a validation against its outlier detection alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [(1, 3), (4, 2, 3), (3, 4)])
def test_batch_of_both(hb, ws, layers):
    pairs, schedules = [], []
    for k, nb in enumerate(layers):
        A, B = hb.synthetic.particle_pair((150, 130 + 10 * k), hb.synthetic.uniform_flow(0.8, -0.6), seed=k, ppp=0.02)
        pairs.append((A, B))
        schedules.append([hb.PIVParameters(window_size=16, overlap=8, n_peaks=3, uod_neighborhood=nb,
                                           validation=(("uod", dict(threshold=3.0, neighborhood_size=5 - nb)),)),
                          hb.PIVParameters(window_size=12, overlap=6, n_peaks=3, uod_neighborhood=nb)])
    for got, (A, B), ps in zip(hb.run_piv_batch(pairs, schedules, workspace=ws), pairs, schedules):
        want = hb.run_piv(A, B, ps, workspace=ws)
        assert want.outliers.any()
        for f in ("u", "v", "outliers"):
            np.testing.assert_array_equal(getattr(got, f), getattr(want, f))


def test_time_of_three_layers(hb, ws):
    from hammerhead_b200 import _lib, hooks

    n, rng = (500, 400), np.random.default_rng(0)
    u, v = rng.normal(0, 0.2, (2,) + n).astype(np.float32)
    wrong = rng.random(n) < 0.01
    u[wrong] += 5 * rng.normal(size=wrong.sum()).astype(np.float32)
    alt = rng.normal(0, 0.2, (2,) + n + (2,)).astype(np.float32)
    p = hb.PIVParameters(window_size=16, overlap=8, uod_neighborhood=3)
    L, prof = _lib.lib(), (_lib.hh_kernel_profile * 5)()

    def device_ms(call):
        best = 1e9
        for _ in range(5):
            _lib.check(L.hh_profile_read(ws.ctx, prof, 1), ws.ctx)
            call()
            _lib.check(L.hh_profile_read(ws.ctx, prof, 1), ws.ctx)
            best = min(best, prof[4].ms)
        return best

    L.hh_set_profiling(ws.ctx, 1)
    try:
        whole = device_ms(lambda: hooks.validate(ws, p, u, v, alt_u=alt[0], alt_v=alt[1], force_replace=True))
        flags = device_ms(lambda: hooks.universal_outlier_detection(ws, u, v, 2.0, 3))
    finally:
        L.hh_set_profiling(ws.ctx, 0)
    assert whole <= 2.0 * flags, (whole, flags)
