"""The adjoint at the edges of its launches' ranges, against the oracle's FP64
loss and analytic gradient (the tolerances of the differentiation case: 1e-5
relative on the loss, 1e-3 relative L2 on dL/dP)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _agrees(hb, orc, ws, A, B, P, grid, window, overlap):
    L, g = hb.NCCLoss(A, B, window=window, overlap=overlap, workspace=ws).value_and_grad(P, grid)
    cA, cB = orc.prefilter(A, dtype=np.float64), orc.prefilter(B, dtype=np.float64)
    wins = orc.ncc_windows(A.shape, window, overlap)
    L64, g64 = orc.ncc_loss_grad(cA, cB, A.shape, P.astype(np.float64), grid, windows=wins, window=window, nthreads=8)
    assert abs(L - L64) <= 1e-5 * abs(L64)
    assert np.linalg.norm(g - g64) <= 1e-3 * np.linalg.norm(g64)


@pytest.mark.parametrize("rows,window,overlap", [(2, 2, 0), (4, 4, 2), (5, 3, 1), (7, 6, 3), (8, 8, 4), (9, 8, 6)])
def test_few_rows(hb, orc, ws, rows, window, overlap):
    """Images with fewer rows than the pixel kernel's block has columns (8)."""
    rng = np.random.default_rng(rows)
    A = rng.random((rows, 61)).astype(np.float32)
    B = (A + 0.2 * rng.random(A.shape)).astype(np.float32)
    P = rng.normal(0.0, 0.2, (2, 9, 2)).astype(np.float32)
    grid = (1.5, rows - 2.0 if rows > 2 else 1.0, 2.0, 7.0)
    _agrees(hb, orc, ws, A, B, P, grid, window, overlap)


def test_wide_image_and_long_node_axis(hb, orc, ws):
    """More column blocks than a grid's second dimension holds (65535): 8 image
    columns and 2 node columns to a block. Displacements are multiples of 1/2 px
    on nodes 4 px apart, so that FP32 holds every sample's coordinate exactly at
    this width."""
    rng = np.random.default_rng(3)
    A = rng.random((8, 524301)).astype(np.float32)
    B = (A + 0.2 * rng.random(A.shape)).astype(np.float32)
    P = (rng.integers(-2, 3, (1, 131075, 2)) / 2).astype(np.float32)
    _agrees(hb, orc, ws, A, B, P, (4.0, 1.0, 2.0, 4.0), 8, 0)


def test_nan_node(hb, orc, ws):
    """A node without a displacement (NaN): the windows it reaches drop out of
    the loss like flat ones, and only its neighbours' gradients are NaN."""
    shape, window, overlap, (i, j) = (90, 101), 16, 8, (3, 4)
    A, B = hb.synthetic.particle_pair(shape, hb.synthetic.uniform_flow(0.7, -0.4), seed=5)
    grid = (8.5, 10.0, 8.5, 11.0)
    P = (np.array([0.7, -0.4]) + np.random.default_rng(5).normal(0.0, 0.3, (8, 9, 2))).astype(np.float32)
    Pn = P.copy()
    Pn[i, j] = np.nan
    L, g = hb.NCCLoss(A, B, window=window, overlap=overlap, workspace=ws).value_and_grad(Pn, grid)
    # pixel rows and columns whose predictor cell has the node as a corner
    cells = [np.clip(np.floor((np.arange(n) + 1.0 - q0) / sp), 0, m - 2)
             for n, q0, sp, m in ((shape[0], 8.5, 10.0, 8), (shape[1], 8.5, 11.0, 9))]
    rows, cols = ((c == k) | (c == k - 1) for c, k in zip(cells, (i, j)))
    wins = orc.ncc_windows(shape, window, overlap)
    hit = np.array([rows[r:r + window].any() and cols[c:c + window].any() for r, c in wins])
    assert 0 < hit.sum() < len(wins)
    cA, cB = orc.prefilter(A, dtype=np.float64), orc.prefilter(B, dtype=np.float64)
    L64, g64 = orc.ncc_loss_grad(cA, cB, shape, P.astype(np.float64), grid, windows=wins[~hit], window=window)
    assert abs(L - L64) <= 1e-5 * abs(L64)
    far = np.ones(P.shape[:2], bool)
    far[i - 1:i + 2, j - 1:j + 2] = False
    assert np.isnan(g[i, j]).all()
    assert np.linalg.norm((g - g64)[far]) <= 1e-3 * np.linalg.norm(g64[far])


def _least_time(call):
    import time

    call()
    times = []
    for _ in range(20):
        t = time.perf_counter()
        call()
        times.append(time.perf_counter() - t)
    return min(times)


def test_small_image_with_many_windows(hb, ws):
    """Some 3900 windows on 92 x 61 pixels share their tiles among as many CTAs
    as on 256 x 256: no more than three times its time (two CTAs took ten)."""
    def loss_time(shape, overlap):
        rng = np.random.default_rng(0)
        A = rng.random(shape).astype(np.float32)
        loss = hb.NCCLoss(A, A[::-1], window=13, overlap=overlap, workspace=ws)
        P, grid = np.zeros((4, 4, 2), np.float32), (7.0, shape[0] / 5, 7.0, shape[1] / 5)
        return _least_time(lambda: loss.value(P, grid))

    assert loss_time((92, 61), 12) <= 3 * loss_time((256, 256), 9)


def test_small_image_gradient(hb, ws):
    """A small image's pixels are dealt over enough threads: with 49 px windows at
    every pixel, loss and gradient take no more than five times the loss (8 columns
    a thread took nine)."""
    rng = np.random.default_rng(0)
    A = rng.random((86, 76)).astype(np.float32)
    loss = hb.NCCLoss(A, A[::-1], window=49, overlap=48, workspace=ws)
    P, grid = np.zeros((20, 20, 2), np.float32), (4.0, 4.0, 4.0, 3.5)
    assert _least_time(lambda: loss.value_and_grad(P, grid)) <= 5 * _least_time(lambda: loss.value(P, grid))
