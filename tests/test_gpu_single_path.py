"""The single-pair call's device grid masks, window lists and result read-back
at their edges: against the host's pass_grid and the batched form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "peak_ratio", "correlation_moment", "uncertainty_u", "uncertainty_v")


@pytest.mark.parametrize("window,search,overlap", [((16, 16), (16, 16), (8, 8)), ((12, 20), (12, 20), (5, 13)),
                                                   ((16, 16), (32, 32), (8, 8)), ((9, 8), (15, 14), (0, 7))])
@pytest.mark.parametrize("thr", [0.01, 0.5, 1.0])
def test_grid_mask_equals_host(hb, ws, window, search, overlap, thr):
    rng = np.random.default_rng(7)
    shape = (83, 101)
    A, B = rng.random((2,) + shape).astype(np.float32)
    mask = np.zeros(shape, bool)
    mask[10:40, 30:70] = True
    mask |= rng.random(shape) < 0.05
    p = hb.PIVParameters(window_size=window, search_area_size=search, overlap=overlap, uncertainty=window == search)
    x, y, gm, _ = hb.pass_grid(shape, p, mask, thr)
    r = hb.run_piv(A, B, p, mask=mask, mask_threshold=thr, workspace=ws)
    np.testing.assert_array_equal(r.mask, gm)
    np.testing.assert_array_equal(r.x, x)
    np.testing.assert_array_equal(r.y, y)
    assert np.isnan(r.u[gm]).all() and np.isnan(r.uncertainty_u[gm]).all()


@pytest.mark.parametrize("smoothing", [True, False])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("side,overlap", [(120, 4), (700, 6)])  # results within and beyond the page-locked block
def test_equals_batched_form(hb, ws, side, overlap, masked, smoothing):
    syn = hb.synthetic
    A, B = syn.particle_pair((side, side + 13), syn.sine_shear_flow(1.5, 150.0), seed=side)
    mask = None
    if masked:
        mask = np.zeros(A.shape, bool)
        mask[20:60, 30:50] = True
    passes = hb.multipass_parameters([16]) + [
        hb.PIVParameters(window_size=8, overlap=overlap, max_iterations=3, uncertainty=True, min_peak_ratio=1.1,
                         validation=(("velocity_magnitude", dict(max=4.0)),))]
    r = hb.run_piv(A, B, passes, mask=mask, predictor_smoothing=smoothing, workspace=ws)
    b = hb.run_piv_batch([(A, B)], passes, masks=[mask], predictor_smoothing=smoothing, workspace=ws)[0]
    for f in FIELDS:
        np.testing.assert_array_equal(getattr(r, f), getattr(b, f), err_msg=f)
    np.testing.assert_array_equal(r.outliers, b.outliers)
