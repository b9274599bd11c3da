"""Deformation strips at the edges of their 32 rows by 8 columns: images of one
strip and less, one past it, ragged sizes, predictor grids of one node on an
axis, samples on and beyond the border. The oracle forms the same sums in the
same order from its own coefficients: 4 ulp of the image scale (1 here), as for
whole images."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 16), (31, 7), (32, 8), (33, 9), (64, 17), (65, 40), (131, 77)])
@pytest.mark.parametrize("nodes", [(1, 1), (1, 3), (4, 1), (3, 5)])
@pytest.mark.parametrize("scale", [0.0, 0.7, 6.0])
def test_strip_edges(ws, orc, shape, nodes, scale):
    from hammerhead_b200 import hooks

    rng = np.random.default_rng(shape[0] * 10 + nodes[1])
    A = rng.uniform(size=shape).astype(np.float32)
    B = rng.uniform(size=shape).astype(np.float32)
    py = (3.5 + np.arange(nodes[0]) * 5).astype(np.float32)
    px = (2.5 + np.arange(nodes[1]) * 2).astype(np.float32)
    pu, pv = (scale * rng.standard_normal((2,) + nodes)).astype(np.float32)
    g = np.array([2.0, 4.0], np.float32)
    sess = hooks.DeviceSession(ws)
    sess.stage_pair(A, B)
    _, _, wA, wB = sess.apply_predictor(pu, pv, py, px, g, g, return_warped=True)
    oA, oB = orc.deform(orc.prefilter(A), orc.prefilter(B), shape, pu, pv, py, px)
    for w, o in ((wA, oA), (wB, oB)):
        assert np.abs(w.astype(np.float64) - o).max() <= 4 * np.spacing(np.float32(1.0))
