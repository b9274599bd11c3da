"""Phase-correlation planes of rectangular and prime lengths against FP64.

A bin enters the plane as w S / (|S| + eps), whose error is at most 2 dS / (|S| +
eps), so the plane's error is bounded by the mean over bins of w min(2, 2 dS / (|S|
+ eps)) and the inverse transform's share. dS comes from the forward transforms'
errors: per bin at most 4 u (log2 P + r) times the norm of the packed frames (u =
2^-24, r the largest prime factor of the lengths, whose direct sum adds a rounding
per term), and in the constant bin the roundings of the means, P u each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _largest_factor(n):
    f, p = 1, 2
    while n > 1:
        while n % p == 0:
            f, n = p, n // p
        p += 1
    return f


@pytest.mark.parametrize("window,search", [((24, 16), None), ((48, 32), None), ((12, 20), None), ((14, 41), None),
                                           ((37, 8), None), ((9, 26), None), ((100, 128), None), ((140, 96), None),
                                           ((16, 12), (24, 30)), ((20, 20), (28, 28)), ((32, 32), (48, 48))])
def test_phase_planes_vs_fp64(hb, ws, window, search):
    from hammerhead_b200 import hooks

    s = search or window
    rng = np.random.default_rng(7 * s[0] + s[1])
    n, m = s[0] + 7, 2 * s[1] + 3
    A = rng.random((n, m)).astype(np.float32)
    B = (np.roll(A, (1, 2), (0, 1)) + 0.3 * rng.random((n, m))).astype(np.float32)
    p = hb.PIVParameters(window_size=window, search_area_size=s, overlap=0, correlation_method="phase")
    jobs = hb.pass_grid((n, m), p)[3]
    d = hooks.DeviceSession(ws)
    d.stage_pair(A, B)
    planes = d.correlation_planes(p, jobs)
    P, u, eps = s[0] * s[1], 2.0 ** -24, float(np.finfo(np.float32).eps)
    fr, fc = (np.fft.fftfreq(k, 1.0 / k) for k in s)
    sigma = min(s) / 8.0
    w = np.exp(-(fr[:, None] ** 2 + fc[None] ** 2) / (2 * sigma ** 2))
    growth = 4 * u * (np.log2(P) + max(_largest_factor(k) for k in s))
    o = [(s[k] - window[k]) // 2 for k in range(2)]
    for j, (_, _, rs, cs) in enumerate(jobs):
        r, c = rs - 1, cs - 1
        a = np.zeros(s)
        x = A[r:r + window[0], c:c + window[1]].astype(float)
        a[o[0]:o[0] + window[0], o[1]:o[1] + window[1]] = x - x.mean()
        b = B[r - o[0]:r - o[0] + s[0], c - o[1]:c - o[1] + s[1]].astype(float)
        mb = b.mean()
        b -= mb
        FA, FB = np.fft.fft2(a), np.fft.fft2(b)
        S = np.conj(FA) * FB
        R = np.fft.fftshift(np.abs(np.fft.ifft2(w * S / (np.abs(S) + eps))))
        if search:
            keep = [np.abs(np.arange(s[k]) - s[k] // 2) <= o[k] for k in range(2)]
            R = R * (keep[0][:, None] & keep[1][None])
        e = np.full(s, growth * np.hypot(np.linalg.norm(a), np.linalg.norm(b)))
        e[0, 0] += P * u * (abs(x.mean()) + abs(mb))
        dS = (np.abs(FA) + np.abs(FB) + e) * e
        bound = np.mean(w * np.minimum(2.0, 2 * dS / (np.abs(S) + eps))) + growth * np.mean(w)
        assert bound < 0.1 * R.max()
        assert np.abs(planes[j] - R).max() <= bound
