"""Quantized growth in rounds on a bag, against growth split by split.

The reference sums the root's packed values by position when it bags, so the
most frequent bin can be left with a negative hessian and the cumulative sums
of a scan need not grow: each threshold's data and hessian minima are tested
in scan order then, as the split-by-split growth's scan (persistent_grow) does.
The bags here are far from the rows' first positions."""
import numpy as np
import pytest

from conftest import binned_dataset

pytestmark = pytest.mark.gpu


def _case(kind, n=20_000, f=10, seed=0):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, f)).astype(np.float32)
    if kind == "missing":  # both directions, with the extra candidate, and zeros as the most frequent bin
        X[rng.random(X.shape) < 0.1] = np.nan
        X[rng.random(X.shape) < 0.3] = 0.0
    z = np.nan_to_num(X[:, 0] + X[:, 1] * X[:, 2])
    y = (rng.random(n) < 1 / (1 + np.exp(-z))).astype(np.float32)
    g = (0.5 - y + 0.3 * rng.standard_normal(n)).astype(np.float32)
    h = (0.1 + 0.2 * rng.random(n)).astype(np.float32)
    if kind == "wide":
        small = rng.random(n) < 0.3
        g[small] = np.ldexp(g[small], -rng.integers(20, 45, int(small.sum())))
        h[::3] = np.ldexp(h[::3], -rng.integers(20, 45, len(h[::3])))
    if kind == "heavy_last":  # the rows past the bag's length weigh more
        h[n // 2:] += 0.2
    return X, y, g, h


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("kind", ["plain", "wide", "heavy_last", "missing"])
def test_bagged_trees_are_those_of_growth_by_split(lgb, kind, seed):
    X, y, g, h = _case(kind, seed=seed)
    n = len(y)
    params = {"objective": "binary", "num_leaves": 31, "num_threads": 4, "seed": 3 + seed, "use_quantized_grad": True,
              "num_grad_quant_bins": 4, "stochastic_rounding": True}
    rng = np.random.default_rng(50 + seed)
    used = np.sort(rng.choice(np.arange(n // 4, n), n // 2, replace=False)).astype(np.uint32)
    ds = binned_dataset(lgb, X, y, params)
    learners = [lgb.Learner(ds, dict(params, persistent_grow=p)) for p in (False, True)]
    trees = []
    for learner in learners:
        learner.set_bagging(used)
        try:
            trees.append(learner.train(g, h)[0])
        except lgb.LightGBMError as e:  # a split without rows on one side: the reference's check
            assert "Check failed" in str(e)
            trees.append(None)
    got, want = trees
    if got is None or want is None:
        assert got is want
        return
    for name in ("num_leaves", "split_feature", "threshold_in_bin", "decision_type", "left_child", "right_child",
                 "leaf_count", "internal_count", "leaf_value", "split_gain_f64"):
        assert np.array_equal(got[name], want[name]), name
