"""Growth in rounds (the default launch strategy) against growth split by split.

The rounds expand many nodes at once and replay the reference's order of
splits afterwards; persistent growth splits one leaf at a time through other
kernels. Both must grow the same trees: quantized form bit for bit, FP64 form
the same splits, rows and leaf values within the FP64 bars (histogram atomics
add in another order)."""
import numpy as np
import pytest

from conftest import binned_dataset

pytestmark = pytest.mark.gpu

CASES = {
    # trees the rounds' bookkeeping ends at: one split, two leaves' worth of rows, no split at all
    "two_leaves": dict(n=500, leaves=2),
    "three_leaves": dict(n=40, leaves=3, p=dict(min_data_in_leaf=5)),
    "no_split": dict(n=300, leaves=31, p=dict(min_data_in_leaf=200, feature_pre_filter=False)),
    "rows_run_out": dict(n=700, leaves=255, p=dict(min_data_in_leaf=3)),
    # row counts around the partition's tile, an odd one, and one feature
    "tile": dict(n=1024, leaves=15, p=dict(min_data_in_leaf=1)),
    "tile_plus_one": dict(n=1025, leaves=15, p=dict(min_data_in_leaf=1)),
    "one_feature": dict(n=20011, leaves=63, f=1),
    # the replay's register form ends at 256 leaves; the explored nodes leave shared memory past 3072
    "leaves_256": dict(n=60000, leaves=256),
    "leaves_257": dict(n=60000, leaves=257),
    "leaves_2500": dict(n=120000, leaves=2500, p=dict(min_data_in_leaf=5)),
    # gain formulas and stopping rules
    "max_depth": dict(n=30000, leaves=63, p=dict(max_depth=5)),
    "l1_delta": dict(n=30000, leaves=31, p=dict(lambda_l1=2.0, max_delta_step=0.4)),
    "smooth": dict(n=30000, leaves=31, p=dict(path_smooth=5.0, min_gain_to_split=0.5)),
    "monotone": dict(n=30000, leaves=31, p=dict(monotone_constraints=[1, -1, 0, 1], monotone_penalty=1.5)),
    "categorical": dict(n=30000, leaves=63, f=40, cats=7),
    "slots": dict(n=20000, leaves=31, k=3, f=33, cats=1),
    "bag": dict(n=30001, leaves=63, bag=True),
    # noise labels: gains hardly fall with depth, so many expansions are never split
    "noise": dict(n=50000, leaves=127, noise=True),
    # a few distinct rows: many exactly equal gains
    "ties": dict(n=4096, leaves=63, ties=True, p=dict(min_data_in_leaf=1)),
}


def _data(n, f=12, cats=0, noise=False, ties=False, seed=0):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, f)).astype(np.float32)
    if f > 4:
        X[rng.random(X.shape) < 0.03] = np.nan
        X[rng.random(X.shape) < 0.1] = 0.0
    if ties:
        X = rng.integers(0, 3, (n, f)).astype(np.float32)
    for j in range(cats):
        X[:, f - 1 - j] = rng.integers(0, 3 + 9 * j, n)
    z = np.nan_to_num(X[:, 0] + X[:, min(1, f - 1)] * X[:, min(2, f - 1)])
    y = rng.random(n) < (0.5 if noise else 1 / (1 + np.exp(-z)))
    return X, y.astype(np.float32)


@pytest.mark.parametrize("form", ["quantized", "f64", "f32c"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_rounds_grow_the_same_trees(lgb, case, form):
    c = CASES[case]
    n, k, f = c["n"], c.get("k", 1), c.get("f", 12)
    cats = list(range(f - c.get("cats", 0), f))
    X, y = _data(n, f, c.get("cats", 0), c.get("noise", False), c.get("ties", False))
    params = {"objective": "binary", "num_leaves": c["leaves"], "num_threads": 4, "seed": 3, **c.get("p", {})}
    if form == "quantized":
        params.update(use_quantized_grad=True, num_grad_quant_bins=4, stochastic_rounding=True)
    else:
        params["hist_precision"] = form
    ds = binned_dataset(lgb, X, y, params, categorical=cats)
    rounds = lgb.Learner(ds, params, num_tree_slots=k)
    steps = lgb.Learner(ds, dict(params, persistent_grow=True), num_tree_slots=k)
    rng = np.random.default_rng(7)
    if c.get("bag"):
        used = np.sort(rng.choice(n, n * 3 // 5, replace=False)).astype(np.uint32)
        rounds.set_bagging(used)
        steps.set_bagging(used)
    for it in range(2):  # the second tree replays the captured graph
        # gradients on a grid, so that FP64 sums are exact in any order
        g = np.round(((0.5 - y) + 0.3 * rng.standard_normal((k, n))) * 1024).astype(np.float32).ravel() / 1024
        h = np.round((0.1 + 0.2 * rng.random((k, n))) * 1024).astype(np.float32).ravel() / 1024
        for slot, (a, b) in enumerate(zip(rounds.train(g, h), steps.train(g, h))):
            assert a["num_leaves"] == b["num_leaves"]
            for name in ("split_feature", "threshold_in_bin", "decision_type", "left_child", "right_child", "leaf_parent",
                         "leaf_count", "leaf_depth", "internal_count", "cat_boundaries", "cat_threshold"):
                assert np.array_equal(a[name], b[name]), name
            for name in ("leaf_value", "leaf_weight", "internal_value", "internal_weight", "split_gain_f64"):
                if form == "quantized":
                    assert np.array_equal(a[name], b[name]), name
                else:
                    np.testing.assert_allclose(a[name], b[name], rtol=1e-9, atol=1e-12, err_msg=name)
            nl = int(a["num_leaves"])
            for u, w in zip(rounds.partition(slot, nl), steps.partition(slot, nl)):
                assert np.array_equal(u, w)
