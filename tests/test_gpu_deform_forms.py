"""Deformation strips of 8, 4 and 2 columns and of row slots (images whose rows
would leave lanes of a strip idle), which only wide images reach, against the
oracle's sums (4 ulp of the image scale, as for the strips' edges); a batch of
both forms against single pairs; and the time of a small image."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(32, 12001), (131, 2411), (64, 3003), (64, 1501), (12, 32007), (33, 12005), (70, 5501),
                                   (4, 60011), (3, 50001), (45, 700)])
def test_forms(ws, orc, shape):
    from hammerhead_b200 import hooks

    rng = np.random.default_rng(shape[0])
    A, B = rng.uniform(size=(2,) + shape).astype(np.float32)
    py = (1.5 + np.arange(3) * shape[0] / 3).astype(np.float32)
    px = (2.5 + np.arange(41) * 8).astype(np.float32)  # most columns lie past the last node, which extends flat
    pu, pv = (1.3 * rng.standard_normal((2, 3, 41))).astype(np.float32)
    g = np.array([2.0, 3.0], np.float32)
    sess = hooks.DeviceSession(ws)
    sess.stage_pair(A, B)
    _, _, wA, wB = sess.apply_predictor(pu, pv, py, px, g, g, return_warped=True)
    oA, oB = orc.deform(orc.prefilter(A), orc.prefilter(B), shape, pu, pv, py, px)
    for w, o in ((wA, oA), (wB, oB)):
        assert np.abs(w.astype(np.float64) - o).max() <= 4 * np.spacing(np.float32(1.0))


@pytest.mark.parametrize("rows", [(40, 64, 129), (96, 128), (21, 200)])
def test_batch_of_both_forms(hb, ws, rows):
    pairs = [hb.synthetic.particle_pair((r, 150), hb.synthetic.uniform_flow(0.8, -0.6), seed=r) for r in rows]
    ps = [hb.PIVParameters(window_size=16, overlap=8, max_iterations=2), hb.PIVParameters(window_size=8, overlap=4)]
    for got, (A, B) in zip(hb.run_piv_batch(pairs, ps, workspace=ws), pairs):
        want = hb.run_piv(A, B, ps, workspace=ws)
        for f in ("u", "v", "peak_ratio", "correlation_moment", "outliers"):
            np.testing.assert_array_equal(getattr(got, f), getattr(want, f))


def test_time_of_a_small_image(hb, ws):
    """100 x 100 pixels take a thread per pixel, not one per strip of 8 columns: a
    third of the time of 1024 x 1024, where the strips' chain is half of it."""
    from hammerhead_b200 import _lib, hooks

    L, prof = _lib.lib(), (_lib.hh_kernel_profile * 5)()
    d = hooks.DeviceSession(ws)
    y = np.array([8.0], np.float32)

    def device_ms(shape):
        A = np.random.default_rng(0).random(shape).astype(np.float32)
        d.stage_pair(A, A)
        p, best = np.full((5, 5), 1.3, np.float32), 1e9
        for _ in range(40):
            _lib.check(L.hh_profile_read(ws.ctx, prof, 1), ws.ctx)
            d.apply_predictor(p, p, 1 + shape[0] / 5 * np.arange(5), 1 + shape[1] / 5 * np.arange(5), y, y)
            _lib.check(L.hh_profile_read(ws.ctx, prof, 1), ws.ctx)
            best = min(best, prof[1].ms)
        return best

    L.hh_set_profiling(ws.ctx, 1)
    try:
        small, large = device_ms((100, 100)), device_ms((1024, 1024))
    finally:
        L.hh_set_profiling(ws.ctx, 0)
    assert small <= 0.46 * large, (small, large)
