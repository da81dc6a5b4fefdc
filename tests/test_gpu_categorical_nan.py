"""Categorical scans whose sort keys or gains are NaN: bins without rows and
cat_smooth=0 (0 / 0), and NaN gradients. The order of the sort stays a
permutation (NaN after the numbers, in bin order) and nothing is indexed by a
split that was never found. Growth in rounds and split by split agree."""
import numpy as np
import pytest

from conftest import binned_dataset

pytestmark = pytest.mark.gpu


def _data(n, seed=0):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, 8)).astype(np.float32)
    for j, cats in ((5, 3), (6, 30), (7, 200)):  # one-hot, and two sorted ones with many rare categories
        X[:, j] = np.minimum(rng.zipf(1.4, n) - 1, cats - 1)
    y = ((X[:, 6] % 3 == 1) ^ (X[:, 0] > 0) ^ (rng.random(n) < 0.2)).astype(np.float32)
    return X, y, rng


def _trees(lgb, params, X, y, g, h):
    ds = binned_dataset(lgb, X, y, params, categorical=[5, 6, 7])
    out = []
    for persistent in (False, True):
        learner = lgb.Learner(ds, dict(params, persistent_grow=persistent))
        out.append([learner.train(g, h)[0] for _ in range(2)])
    return out


def _params(form, leaves):
    p = {"objective": "binary", "num_leaves": leaves, "min_data_in_leaf": 3, "min_sum_hessian_in_leaf": 0.0,
         "lambda_l2": 1.0, "cat_smooth": 0.0, "min_data_per_group": 1, "num_threads": 4, "seed": 2}
    if form == "quantized":
        p.update(use_quantized_grad=True, num_grad_quant_bins=16, stochastic_rounding=True)
    else:
        p["hist_precision"] = form
    return p


@pytest.mark.parametrize("form", ["quantized", "f64", "f32c"])
@pytest.mark.parametrize("n,leaves", [(900, 200), (20_000, 127)])
def test_empty_categories_without_smoothing(lgb, form, n, leaves):
    X, y, rng = _data(n)
    # on a grid, so that FP64 sums are exact in any order
    g = np.round((0.5 - y + 0.2 * rng.standard_normal(n)) * 256).astype(np.float32) / 256
    h = np.round((0.1 + 0.2 * rng.random(n)) * 256).astype(np.float32) / 256
    rounds, steps = _trees(lgb, _params(form, leaves), X, y, g, h)
    for a, b in zip(rounds, steps):
        for name in ("num_leaves", "split_feature", "threshold_in_bin", "decision_type", "leaf_count", "cat_boundaries",
                     "cat_threshold"):
            assert np.array_equal(a[name], b[name]), name
        assert (np.asarray(a["decision_type"]) & 1).any()


@pytest.mark.parametrize("form", ["quantized", "f64", "f32c"])
@pytest.mark.parametrize("share", [0.001, 1.0])
def test_nan_gradients(lgb, form, share):
    n = 5000
    X, y, rng = _data(n)
    g = (0.5 - y).astype(np.float32)
    g[rng.random(n) < share] = np.nan
    rounds, steps = _trees(lgb, _params(form, 31), X, y, g, np.full(n, 0.25, np.float32))
    for a, b in zip(rounds, steps):
        assert a["num_leaves"] == b["num_leaves"]
        assert np.array_equal(a["split_feature"], b["split_feature"])
