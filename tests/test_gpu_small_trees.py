"""Quantized trees of few leaves grow split by split, in three launches a split
(a round costs more than the few splits it saves), larger ones in rounds; both
sides of the rule against persistent growth, bit for bit."""
import numpy as np
import pytest

from conftest import binned_dataset

pytestmark = pytest.mark.gpu

# features, tree slots, most leaves of growth split by split
RULE = [(12, 1, 18), (150, 1, 18), (151, 1, 10), (12, 2, 12), (160, 3, 12), (12, 4, 8), (12, 6, 0)]


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("f,k,few", RULE)
def test_few_leaves(lgb, f, k, few, graph):
    rng = np.random.default_rng(f + k)
    n = 20_011
    X = rng.standard_normal((n, f)).astype(np.float32)
    X[rng.random(X.shape) < 0.03] = np.nan
    X[:, f - 1] = rng.integers(0, 12, n)
    X[:, f - 2] = rng.integers(0, 3, n)
    y = (rng.random(n) < 1 / (1 + np.exp(-np.nan_to_num(X[:, 0] + X[:, 1] * X[:, 2])))).astype(np.float32)
    base = {"objective": "binary", "num_threads": 4, "seed": 3, "use_quantized_grad": True, "num_grad_quant_bins": 4,
            "stochastic_rounding": True, "quant_train_renew_leaf": True, "use_cuda_graph": graph}
    ds = binned_dataset(lgb, X, y, base, categorical=[f - 2, f - 1])
    for leaves in sorted({2, 3, max(2, few), few + 1 if few else 4}):
        params = dict(base, num_leaves=leaves)
        one, steps = lgb.Learner(ds, params, num_tree_slots=k), lgb.Learner(ds, dict(params, persistent_grow=True), num_tree_slots=k)
        used = np.sort(rng.choice(n, n // 2, replace=False)).astype(np.uint32)
        for it in range(3):  # the second replays the captured graph, the third is bagged
            if it == 2:
                one.set_bagging(used)
                steps.set_bagging(used)
            g = (0.5 - y + 0.3 * rng.standard_normal((k, n))).astype(np.float32).ravel()
            h = (0.1 + 0.2 * rng.random(k * n)).astype(np.float32)
            got, want = [], []
            for learner, out in ((one, got), (steps, want)):
                try:
                    out.extend(learner.train(g, h))
                except lgb.LightGBMError as e:  # a split without rows on one side: the reference's check
                    assert "Check failed" in str(e)
            if not got or not want:
                assert got == want
                continue
            for slot, (a, b) in enumerate(zip(got, want)):
                for name in a:
                    assert np.array_equal(a[name], b[name]), name
                nl = int(a["num_leaves"])
                for u, w in zip(one.partition(slot, nl), steps.partition(slot, nl)):
                    assert np.array_equal(u, w)
            if leaves <= few:  # the root, three launches a split, the last split's end, the leaves' renewal
                assert one.last_timing()[2] == 1 + 3 * (leaves - 1) + 1 + 2
        one = lgb.Learner(ds, params, num_tree_slots=k)
        one.set_timing(True)
        one.train(g, h)
        if leaves <= few:
            assert len(one.step_times()) == leaves - 1


OPTIONS = {
    "l1_delta": dict(lambda_l1=2.0, max_delta_step=0.4), "smooth": dict(path_smooth=5.0, min_gain_to_split=0.5),
    "monotone": dict(monotone_constraints=[1, -1, 0, 1], monotone_penalty=1.5), "max_depth": dict(max_depth=3),
    "no_split": dict(min_data_in_leaf=2500, feature_pre_filter=False), "rows_run_out": dict(min_data_in_leaf=600),
    "no_renewal": dict(quant_train_renew_leaf=False), "many_bins": dict(num_grad_quant_bins=32),
}


@pytest.mark.parametrize("option", sorted(OPTIONS))
def test_options(lgb, option):
    """The other rules of growth, a feature mask and data-parallel growth (one rank) of a learner of few leaves."""
    rng = np.random.default_rng(9)
    n, f = 4099, 12
    X = rng.standard_normal((n, f)).astype(np.float32)
    X[rng.random(X.shape) < 0.05] = 0.0
    y = (X[:, 0] + X[:, 1] * X[:, 2] + 0.5 * rng.standard_normal(n) > 0).astype(np.float32)
    params = {"objective": "binary", "num_leaves": 15, "num_threads": 4, "seed": 3, "use_quantized_grad": True,
              "num_grad_quant_bins": 4, "stochastic_rounding": True, "quant_train_renew_leaf": True, **OPTIONS[option]}
    ds = binned_dataset(lgb, X, y, params)
    one, parallel = lgb.Learner(ds, params), lgb.Learner(ds, params)
    steps = lgb.Learner(ds, dict(params, persistent_grow=True))
    parallel.set_data_parallel(0, n, lambda ptr, count, dtype, op: None)
    mask = np.ones(ds.binned()["num_features"], np.uint8)
    for it in range(3):
        if it == 2:
            mask[::2] = 0
            for learner in (one, parallel, steps):
                learner.set_feature_mask(0, mask)
        g = (0.5 - y + 0.3 * rng.standard_normal(n)).astype(np.float32)
        h = (0.1 + 0.2 * rng.random(n)).astype(np.float32)
        a, b, c = (learner.train(g, h)[0] for learner in (one, parallel, steps))
        for name in a:
            assert np.array_equal(a[name], c[name]), name
        for name in ("num_leaves", "split_feature", "threshold_in_bin", "leaf_count"):
            assert np.array_equal(b[name], c[name]), name
