"""Categorical splits whose sorted scan takes more than one warp's width of
positions (max_cat_threshold above 32), small groups and both directions,
against the oracle's trees."""
import numpy as np
import pytest

from conftest import binned_dataset, within

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["f64", "quantized"])
@pytest.mark.parametrize("cats,threshold,group", [(60, 32, 100), (66, 33, 10), (200, 64, 1), (240, 200, 30)])
def test_wide_categorical_splits_match_oracle(lgb, orc, form, cats, threshold, group):
    rng = np.random.default_rng(cats)
    n = 30_000
    X = rng.standard_normal((n, 6)).astype(np.float32)
    X[:, 4] = rng.integers(0, cats, n)
    X[:, 5] = np.minimum(rng.geometric(0.05, n), cats - 1)
    effect = rng.standard_normal(cats)
    g = (effect[X[:, 4].astype(int)] + 0.3 * X[:, 0] + 0.5 * rng.standard_normal(n))
    g = (np.round(g * 256) / 256).astype(np.float32)
    h = np.full(n, 0.25, np.float32)
    params = {"objective": "binary", "num_leaves": 15, "max_cat_threshold": threshold, "min_data_per_group": group,
              "cat_smooth": 5.0, "max_cat_to_onehot": 4, "num_threads": 4, "seed": 1}
    if form == "quantized":
        params.update(use_quantized_grad=True, num_grad_quant_bins=4, stochastic_rounding=True)
    ds = binned_dataset(lgb, X, (g > 0).astype(np.float32), params, categorical=[4, 5])
    a = lgb.Learner(ds, params).train(g, h)[0]
    o = orc.train_trees(lgb.resolve_params(params), ds.binned(), g, h).trees[0]
    assert a["num_leaves"] == o["num_leaves"]
    assert a["num_cat"] > 0
    for name in ("split_feature", "threshold_in_bin", "decision_type", "left_child", "right_child", "leaf_count",
                 "cat_boundaries", "cat_threshold"):
        assert np.array_equal(a[name], o[name]), name
    assert within(a["leaf_value"], o["leaf_value"], "leaf_value")
