"""The peak paths of the fused correlation kernels against the plane analysis.

process_windows ranks the peaks inside the correlation kernel (from the row
maxima of an unpadded plane, by column strips of the box of a padded one);
correlation_planes + analyze_planes ranks them from the whole plane, pixel by
pixel. Both see the same plane, so peaks and refined values are the same bit
for bit, at every FFT size, for ties (quantised and constant images), planes
with fewer regional maxima than peaks asked for, and windows holding NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _image(kind, n, rng):
    if kind == "noise":
        return rng.random((n, n)), rng.random((n, n))
    if kind == "steps":  # few grey levels: equal values all over the plane
        a = rng.integers(0, 2, (n, n)).astype(float)
        return a, np.roll(a, (2, 3), (0, 1))
    if kind == "stripes":  # rows of the plane repeat: no row maximum stands out
        a = np.tile((np.arange(n) % 4 == 0).astype(float), (n, 1))
        return a, a
    a = np.zeros((n, n))  # flat except for one speck, and a NaN and an Inf pixel
    b = a.copy()
    a[n // 3, n // 3] = b[n // 3 + 1, n // 3 + 2] = 1.0
    a[5, 5], b[n - 6, 7] = np.nan, np.inf
    return a, b


@pytest.mark.parametrize("padding", [False, True])
@pytest.mark.parametrize("fft", [16, 24, 32, 48, 64, 96, 128])
def test_peaks_equal_plane_analysis(fft, padding):
    import hammerhead_b200 as hb
    from hammerhead_b200 import hooks

    w = fft // 2 if padding else fft
    n = 3 * w + 5  # a ragged grid: several windows per CTA, a part-empty last one
    rng = np.random.default_rng(fft + padding)
    with hb.piv_workspace() as ws:
        d = hooks.DeviceSession(ws)
        for kind in ("noise", "steps", "stripes", "speck"):
            A, B = _image(kind, n, rng)
            d.stage_pair(A.astype(np.float32), B.astype(np.float32))
            for n_peaks, finder, apod, search in ((3, "regionalmax", "gauss", w), (8, "regionalmax", "none", w),
                                                  (4, "exclusion", "none", w), (3, "regionalmax", "none", w - 6)):
                if search != w and padding:
                    continue
                p = hb.PIVParameters(window_size=search, search_area_size=w, overlap=search // 2, padding=padding,
                                     apodization=apod, n_peaks=n_peaks, peak_finder=finder)
                _, _, _, jobs = hb.pass_grid((n, n), p)
                out, locs, _ = d.process_windows(p, jobs, want_locs=True)
                ref, rlocs = hooks.analyze_planes(ws, d.correlation_planes(p, jobs), n_peaks, finder)
                np.testing.assert_array_equal(locs, rlocs, err_msg=f"{kind} {n_peaks} {finder} {apod} {search}")
                np.testing.assert_array_equal(out, ref, err_msg=f"{kind} {n_peaks} {finder} {apod} {search}")


@pytest.mark.parametrize("method", ["cross", "phase"])
@pytest.mark.parametrize("padding", [False, True])
@pytest.mark.parametrize("fft", [16, 32, 48, 64])
def test_default_equals_alternative_shape(fft, padding, method):
    """The default kernel of a class against its alternative CTA shape
    (variant 1, the same arithmetic on another thread mapping), with an image
    mask, partly and fully masked windows, and a part-empty last unit: planes,
    peaks and packed scalars bit for bit."""
    import hammerhead_b200 as hb
    from hammerhead_b200 import hooks

    w = fft // 2 if padding else fft
    n, m = 5 * w + 3, 4 * w + 1
    rng = np.random.default_rng(fft)
    A, B = rng.random((2, n, m)).astype(np.float32)
    mask = np.zeros((n, m), np.uint8)
    mask[: w + w // 2, : 2 * w] = 1
    mask[rng.integers(0, n, 40), rng.integers(0, m, 40)] = 1
    p = hb.PIVParameters(window_size=w, overlap=w // 4, padding=padding, correlation_method=method, apodization="gauss")
    _, _, _, jobs = hb.pass_grid((n, m), p)
    got = []
    with hb.piv_workspace() as ws:
        d = hooks.DeviceSession(ws)
        d.stage_pair(A, B)
        for use in (None, mask):
            d.stage_mask(use)
            for v in (0, 1):
                hb.tuning.set_variant(ws, fft, w, v)
                got.append(d.process_windows(p, jobs[:-1], want_locs=True)[:2] + (d.correlation_planes(p, jobs[:-1]),))
    for k in (0, 2):
        for x, y in zip(got[k], got[k + 1]):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("window,search", [((24, 16), None), ((48, 32), None), ((12, 20), None), ((14, 22), None),
                                           ((9, 26), None), ((64, 4), None), ((4, 34), None), ((50, 10), None),
                                           ((128, 40), None), ((16, 12), (24, 30)), ((100, 128), None)])
@pytest.mark.parametrize("method", ["cross", "phase"])
def test_general_shapes_vs_fp64(window, search, method):
    """General shapes (prime factors 2 to 17, register and Stockham lengths,
    planes for every CTA size): the unpadded plane against numpy in FP64
    (within 2e-5 of the peak), and the peaks against the plane analysis, bit for bit."""
    import hammerhead_b200 as hb
    from hammerhead_b200 import hooks

    s = search or window
    rng = np.random.default_rng(sum(window))
    n, m = s[0] + 7, 2 * s[1] + 3
    A, B = rng.random((2, n, m)).astype(np.float32)
    p = hb.PIVParameters(window_size=window, search_area_size=s, overlap=0, correlation_method=method, n_peaks=4)
    _, _, _, jobs = hb.pass_grid((n, m), p)
    with hb.piv_workspace() as ws:
        d = hooks.DeviceSession(ws)
        d.stage_pair(A, B)
        planes = d.correlation_planes(p, jobs)
        out, locs, _ = d.process_windows(p, jobs, want_locs=True)
        if s[0] * s[1] * 4 <= 180 * 1024:
            ref, rlocs = hooks.analyze_planes(ws, planes, 4)
            np.testing.assert_array_equal(locs, rlocs)
            np.testing.assert_array_equal(out, ref)
    if method == "phase":  # bins of small magnitude: no bound on the plane by its peak
        return
    o = [(s[k] - window[k]) // 2 for k in range(2)]
    for j, (_, _, rs, cs) in enumerate(jobs):
        r, c = rs - 1, cs - 1
        a = np.zeros(s)
        w = A[r:r + window[0], c:c + window[1]].astype(float)
        a[o[0]:o[0] + window[0], o[1]:o[1] + window[1]] = w - w.mean()
        b = B[r - o[0]:r - o[0] + s[0], c - o[1]:c - o[1] + s[1]].astype(float)
        S = np.conj(np.fft.fft2(a)) * np.fft.fft2(b - b.mean())
        R = np.fft.fftshift(np.abs(np.fft.ifft2(S)))
        if search:
            keep = [np.abs(np.arange(s[k]) - s[k] // 2) <= o[k] for k in range(2)]
            R = R * (keep[0][:, None] & keep[1][None])
        assert np.abs(planes[j] - R).max() <= 2e-5 * R.max()


@pytest.mark.parametrize("n_peaks", [1, 2, 4, 8])
def test_epilogue_split_and_whole(ws, hb, n_peaks):
    """A thread per window and peak below 32768 windows, one per window above:
    the same windows through both, every packed value alike."""
    from hammerhead_b200 import hooks, synthetic

    A, B = synthetic.particle_pair((420, 400), synthetic.uniform_flow(1.4, -0.8), seed=21, ppp=0.02)
    A[100:140, 100:140] = B[100:140, 100:140] = 0.25  # windows without a peak
    p = hb.PIVParameters(window_size=16, overlap=14, padding=False, apodization="none", n_peaks=n_peaks)
    jobs = hb.pass_grid(A.shape, p)[3]
    jobs = np.concatenate([jobs, jobs[:: -1]])
    assert len(jobs) > 32768
    sess = hooks.DeviceSession(ws)
    sess.stage_pair(A, B)
    whole, wlocs, _ = sess.process_windows(p, jobs, want_locs=True)
    for i in (0, len(jobs) // 2, len(jobs) - 1000):
        part, plocs, _ = sess.process_windows(p, jobs[i:i + 1000], want_locs=True)
        np.testing.assert_array_equal(part, whole[i:i + 1000])
        np.testing.assert_array_equal(plocs, wlocs[i:i + 1000])
