"""The float forms' histograms in exact fixed point: gradients of few and of many
binary orders of magnitude (two and three limbs a value, and the ranges past
them that keep FP64 adds), constant and zero hessians, more rows than a cell
takes between flushes. A leaf's weight is its hessian sum, taken from the
histograms of its ancestors: it must equal the exact sum of its rows, and the
tree the one grown split by split with FP64 adds."""
import math

import numpy as np
import pytest

from conftest import binned_dataset

pytestmark = pytest.mark.gpu

KINDS = ["two_limbs", "three_limbs", "too_wide", "constant", "zeros", "denormal", "wide_hessian"]


def _grads(kind, y, rng):
    n = len(y)
    g = (0.5 - y + 0.2 * rng.standard_normal(n)).astype(np.float32)
    h = (0.1 + 0.15 * rng.random(n)).astype(np.float32)
    small = rng.random(n) < 0.3
    if kind == "three_limbs":
        g[small] *= np.float32(2.0**-28)
    elif kind == "too_wide":
        g[small] *= np.float32(2.0**-60)
    elif kind == "constant":
        h[:] = np.float32(0.7)
    elif kind == "zeros":
        g[small] = 0.0
        h[small] = 0.0
    elif kind == "denormal":
        g[small] = np.float32(1e-41)
    elif kind == "wide_hessian":
        h[small] *= np.float32(2.0**-25)
    return g, h


@pytest.mark.parametrize("form", ["f64", "f32c"])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,f", [(900, 5), (300_000, 40)])
def test_leaf_weights_are_exact_sums(lgb, kind, form, n, f):
    rng = np.random.default_rng(5)
    X = rng.standard_normal((n, f)).astype(np.float32)
    X[:, 3] = np.round(X[:, 3])  # few bins: most rows of a CTA in a few cells
    y = (X[:, 0] + X[:, 1] * X[:, 2] + 0.5 * rng.standard_normal(n) > 0).astype(np.float32)
    params = {"objective": "binary", "num_leaves": 31, "hist_precision": form, "num_threads": 4}
    ds = binned_dataset(lgb, X, y, params)
    rounds, steps = lgb.Learner(ds, params), lgb.Learner(ds, dict(params, persistent_grow=True))
    g, h = _grads(kind, y, rng)
    a, b = rounds.train(g, h)[0], steps.train(g, h)[0]
    for name in ("num_leaves", "split_feature", "threshold_in_bin", "leaf_count"):
        assert np.array_equal(a[name], b[name]), name
    for name in ("leaf_value", "leaf_weight", "split_gain_f64"):
        # the bars of FP64 sums in another order; the compensated form's FP32 pairs are nearer 1e-7
        np.testing.assert_allclose(a[name], b[name], rtol=1e-9 if form == "f64" else 1e-6, atol=1e-12, err_msg=name)
    begin, count, rows = rounds.partition(0, int(a["num_leaves"]))
    for leaf in range(int(a["num_leaves"])):
        # FP64 sums of up to n rows of at most 1 in histograms, then of up to 255 bins: n * 2^-53 * 255 at the very most
        want = math.fsum(h[rows[begin[leaf]:begin[leaf] + count[leaf]]].astype(np.float64))
        assert abs(a["leaf_weight"][leaf] - want) <= 1e-11 * max(want, 1.0), (leaf, a["leaf_weight"][leaf], want)
