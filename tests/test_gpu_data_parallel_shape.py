"""The data-parallel learner's launches: those of growth split by split, not
of the rounds the learner was created for, and on many features the quantized
scans a warp each. One rank, whose reductions are the identity."""
import numpy as np
import pytest

from conftest import binned_dataset

pytestmark = pytest.mark.gpu


def _case(lgb, form, f, cats, n=20_000, leaves=31):
    rng = np.random.default_rng(3)
    X = rng.standard_normal((n, f)).astype(np.float32)
    X[rng.random(X.shape) < 0.03] = np.nan
    for j in range(cats):
        X[:, f - 1 - j] = rng.integers(0, 4 + 30 * j, n)
    z = np.nan_to_num(X[:, 0] + X[:, 1] * X[:, 2])
    y = (rng.random(n) < 1 / (1 + np.exp(-z))).astype(np.float32)
    params = {"objective": "binary", "num_leaves": leaves, "num_threads": 4, "seed": 3}
    if form == "quantized":
        params.update(use_quantized_grad=True, num_grad_quant_bins=4, stochastic_rounding=True)
    else:
        params["hist_precision"] = form
    ds = binned_dataset(lgb, X, y, params, categorical=list(range(f - cats, f)))
    return ds, params, y, rng


def _parallel(learner, n):
    learner.set_data_parallel(0, n, lambda ptr, count, dtype, op: None)
    return learner


@pytest.mark.parametrize("form", ["quantized", "f64", "f32c"])
def test_grids_of_split_steps(lgb, form):
    ds, params, y, _ = _case(lgb, form, 12, 0)
    steps = lgb.Learner(ds, dict(params, persistent_grow=True)).launch_shape
    assert _parallel(lgb.Learner(ds, params), len(y)).launch_shape == steps
    # a shape the caller chose stays
    chosen = {"partition_ctas": 77, "hist_ctas": 64, "hist_rows_per_block": 1024}
    learner = lgb.Learner(ds, params)
    learner.launch_shape = chosen
    assert _parallel(learner, len(y)).launch_shape == chosen


# features around a warp's and a launch's share of scans, and where the block scans end
@pytest.mark.parametrize("f", [3, 148, 149, 300, 1200])
def test_scans_by_warp_grow_the_same_trees(lgb, f):
    ds, params, y, rng = _case(lgb, "quantized", f, 3 if f > 3 else 0)
    one, parallel = lgb.Learner(ds, params), _parallel(lgb.Learner(ds, params), len(y))
    for it in range(2):
        g = (0.5 - y + 0.3 * rng.standard_normal(len(y))).astype(np.float32)
        h = (0.1 + 0.2 * rng.random(len(y))).astype(np.float32)
        a, b = one.train(g, h)[0], parallel.train(g, h)[0]
        for name in ("num_leaves", "split_feature", "threshold_in_bin", "decision_type", "leaf_count", "leaf_value",
                     "split_gain_f64", "cat_threshold"):
            assert np.array_equal(a[name], b[name]), name


@pytest.mark.parametrize("form", ["quantized", "f64", "f32c"])
def test_wide_scans_grow_the_same_trees(lgb, monkeypatch, form):
    """Both scans of a split step (LGBM_B200_SCAN_WIDE: the 256-thread scan with
    one CTA an SM; the register-capped one, or, quantized, a warp a scan), which
    data-parallel growth alone launches, on numerical and categorical features
    with missing values, and the rounds' scan."""
    ds, params, y, rng = _case(lgb, form, 20, 3)
    learners = [lgb.Learner(ds, params)]
    for wide in "01":
        monkeypatch.setenv("LGBM_B200_SCAN_WIDE", wide)
        learners.append(_parallel(lgb.Learner(ds, params), len(y)))
    categorical = False
    for it in range(2):
        # on a grid, so that FP64 sums are exact in any order
        g = np.round((0.5 - y + 0.3 * rng.standard_normal(len(y))) * 1024).astype(np.float32) / 1024
        h = np.round((0.1 + 0.2 * rng.random(len(y))) * 1024).astype(np.float32) / 1024
        rounds, narrow, wide = (learner.train(g, h)[0] for learner in learners)
        for name in ("num_leaves", "split_feature", "threshold_in_bin", "decision_type", "leaf_count", "cat_threshold"):
            assert np.array_equal(narrow[name], wide[name]), name
            assert np.array_equal(narrow[name], rounds[name]), name
        categorical |= bool((np.asarray(narrow["decision_type"]) & 1).any())
    assert categorical
