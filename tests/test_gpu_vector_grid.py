"""Vector-grid kernels where a cell's route or a grid's split can go wrong:
substitution and replacement with full, partial and empty neighbourhoods of
each size (1 and 2 layers in registers, 3 in indexed arrays; a hole whose first
square is short of 3 donors), and the convergence norm at grids of less than a
warp up to several rounds of the cluster, with ties, none and few counted
cells. Identical inputs must give the oracle's values exactly."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hooks():
    from hammerhead_b200 import hooks

    return hooks


def _field(rng, shape, spikes):
    u = (2.0 + 0.1 * rng.standard_normal(shape)).astype(np.float32)
    v = (-1.0 + 0.1 * rng.standard_normal(shape)).astype(np.float32)
    at = rng.uniform(size=shape) < spikes
    u[at] += rng.uniform(-8, 8, int(at.sum())).astype(np.float32)
    v[at] += rng.uniform(-8, 8, int(at.sum())).astype(np.float32)
    u.flat[:: 11] = u.flat[0]  # ties
    return u, v


@pytest.mark.parametrize("shape", [(1, 1), (1, 9), (2, 2), (5, 3), (31, 40)])
@pytest.mark.parametrize("nb", [1, 2, 3])
@pytest.mark.parametrize("spikes", [0.02, 0.4])
def test_substitution_and_replacement(ws, orc, hb, hooks, shape, nb, spikes):
    rng = np.random.default_rng(100 * nb + shape[1])
    u, v = _field(rng, shape, spikes)
    ratio = np.where(rng.uniform(size=shape) < spikes, 1.0, 2.0).astype(np.float32)
    u[rng.uniform(size=shape) < 0.02] = np.nan
    au = (2.0 + 0.3 * rng.standard_normal(shape + (2,))).astype(np.float32)
    av = (-1.0 + 0.3 * rng.standard_normal(shape + (2,))).astype(np.float32)
    mask = rng.uniform(size=shape) < 0.05
    mask[: shape[0] // 3, : shape[1] // 3] = shape[0] > 8  # a masked corner
    p = hb.PIVParameters(uod_neighborhood=nb, min_peak_ratio=1.5, replace_outliers=True)
    got = hooks.validate(ws, p, u, v, ratio, np.zeros_like(u), mask, au, av)
    want = orc.validate(p, u, v, ratio, np.zeros_like(u), mask, au, av)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("shape,share", [((1, 1), 1.0), ((2, 2), 0.5), ((1, 17), 0.6), ((33, 29), 0.1), ((33, 29), 0.8),
                                         ((40, 37), 0.97), ((9, 9), 1.0)])
def test_replacement_holes(ws, orc, hooks, shape, share):
    rng = np.random.default_rng(7 + shape[0])
    u, v = _field(rng, shape, 0.0)
    u[rng.uniform(size=shape) < 0.03] = np.nan
    inv = rng.uniform(size=shape) < share
    got = hooks.replace_vectors(ws, u, v, inv)
    want = orc.replace_vectors(u, v, inv, dtype=np.float32)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 225, 4095, 4097, 70001])
@pytest.mark.parametrize("kind", ["random", "ties", "spread", "masked", "one"])
def test_convergence_norm(ws, orc, hooks, n, kind):
    rng = np.random.default_rng(n)
    pu, pv = rng.standard_normal((2, n)).astype(np.float32)
    step = {"ties": np.float32(0.25) * rng.integers(0, 3, (2, n)), "spread": 10.0 ** rng.uniform(-12, 6, (2, n))}
    d = step.get(kind, 0.01 * rng.standard_normal((2, n))).astype(np.float32)
    if kind == "ties":
        pu, pv = np.zeros((2, n), np.float32)
    u, v = pu + d[0], pv + d[1]
    u[n // 2:: 97] = np.nan
    m = np.zeros(n, bool)
    if kind == "masked":
        m[:] = True
    if kind == "one":
        m[:] = True
        m[n - 1] = False
    a, b = hooks.field_change(ws, u, v, pu, pv, m), orc.field_change(u, v, pu, pv, m)
    assert a == b or (math.isnan(a) and math.isnan(b))
