"""The adjoint's tiles at their edges: window sizes with one and several
windows per tile, overlaps from none to all but one pixel, ragged frames,
predictor grids coarser and finer than the windows, and single-node axes,
against the oracle's FP64 loss and analytic gradient (the tolerances of the
differentiation case: 1e-5 relative on the loss, 1e-3 relative L2 on dL/dP)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,window,overlap,nodes", [
    ((70, 83), 16, 8, (7, 9)), ((131, 97), 8, 0, (17, 33)), ((90, 75), 12, 11, (2, 1)), ((101, 140), 24, 12, (1, 8)),
    ((129, 66), 32, 16, (40, 21)), ((97, 160), 48, 40, (5, 5)), ((130, 200), 64, 32, (9, 14)), ((64, 64), 64, 0, (3, 3))])
def test_shapes_vs_fp64(hb, orc, ws, shape, window, overlap, nodes):
    syn = hb.synthetic
    A, B = syn.particle_pair(shape, syn.uniform_flow(0.7, -0.4), seed=window + overlap)
    rng = np.random.default_rng(window)
    ysp = max((shape[0] - window) / max(nodes[0] - 1, 1), 1.5)
    xsp = max((shape[1] - window) / max(nodes[1] - 1, 1), 1.5)
    grid = (window / 2 + 0.5, ysp, window / 2 + 0.5, xsp)
    P = (np.array([0.7, -0.4]) + rng.normal(0.0, 0.3, nodes + (2,))).astype(np.float32)
    L, g = hb.NCCLoss(A, B, window=window, overlap=overlap, workspace=ws).value_and_grad(P, grid)
    cA, cB = orc.prefilter(A, dtype=np.float64), orc.prefilter(B, dtype=np.float64)
    wins = orc.ncc_windows(shape, window, overlap)
    L64, g64 = orc.ncc_loss_grad(cA, cB, shape, P.astype(np.float64), grid, windows=wins, window=window, nthreads=8)
    assert abs(L - L64) <= 1e-5 * abs(L64)
    assert np.linalg.norm(g - g64) <= 1e-3 * np.linalg.norm(g64)
