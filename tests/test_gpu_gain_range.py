"""Gains at the edge of FP32's range. The scans of a growth round leave out
thresholds by an FP32 estimate of their gain; with gradients and hessian sums
so small (or large) that the estimate loses its precision while its value looks
ordinary, the trees must still be those of FP64 gains (growth split by split)."""
import numpy as np
import pytest

from conftest import binned_dataset

pytestmark = pytest.mark.gpu

# binary orders of the gradients and hessians
SCALES = {
    "denormal_squares": (-73, -48),  # squares of sums below 2^-126 over hessian sums of about 1e-13: gains of about 1e-29
    "rows_near_epsilon": (-74, -60),  # a row's hessian near the reference's epsilon of 1e-15
    "rows_below_epsilon": (-76, -66),
    "huge_hessians": (60, 114),      # divisors around 2^126
    "largest": (60, 100),
    "ordinary": (0, 0),
}


@pytest.mark.parametrize("form", ["f64", "f32c", "quantized"])
@pytest.mark.parametrize("scale", sorted(SCALES))
def test_trees_are_those_of_fp64_gains(lgb, scale, form):
    rng = np.random.default_rng(8)
    n, f = 20_000, 20
    X = rng.standard_normal((n, f)).astype(np.float32)
    params = {"objective": "regression", "num_leaves": 127, "min_data_in_leaf": 5, "min_sum_hessian_in_leaf": 0.0,
              "num_threads": 4, "seed": 1}
    if form == "quantized":
        params.update(use_quantized_grad=True, num_grad_quant_bins=32, stochastic_rounding=True)
    else:
        params["hist_precision"] = form
    ds = binned_dataset(lgb, X, X[:, 0], params)
    rounds, steps = lgb.Learner(ds, params), lgb.Learner(ds, dict(params, persistent_grow=True))
    sg, sh = (np.float32(2.0) ** np.float32(e) for e in SCALES[scale])
    for it in range(3):
        # noise on a grid, so that FP64 sums are exact in any order: many thresholds of nearly the same gain
        g = np.round(rng.standard_normal(n) * 256).astype(np.float32) / 256 * sg
        h = np.round((0.5 + 0.5 * rng.random(n)) * 256).astype(np.float32) / 256 * sh
        trees = []
        for learner in (rounds, steps):
            try:
                trees.append(learner.train(g, h)[0])
            except lgb.LightGBMError as e:  # row counts estimated from the hessians left a side without rows
                assert "Check failed" in str(e)
                trees.append(None)
        a, b = trees
        if a is None or b is None:
            assert a is b
            continue
        for name in ("num_leaves", "split_feature", "threshold_in_bin", "leaf_count"):
            assert np.array_equal(a[name], b[name]), name
