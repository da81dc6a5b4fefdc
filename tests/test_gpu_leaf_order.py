"""What a leaf gives does not depend on how far the rounds expanded it.

A leaf expanded past the finished tree loses its row list to its descendants'.
Renewed leaf values are sums over that list, so rounds and growth split by
split (persistent_grow, whose lists are never lost) must give the same bits
from gradients that an FP64 sum rounds in every order; and the partition's
readback must give the lists in their own order."""
import numpy as np
import pytest

from conftest import binned_dataset

pytestmark = pytest.mark.gpu

CASES = {
    "plain": dict(n=40_003, leaves=63),
    # gains that hardly fall with depth: many expansions the finished tree has no use for, several levels deep
    "noise": dict(n=60_001, leaves=127, noise=True),
    "slots": dict(n=20_000, leaves=31, k=3, noise=True),
    "bag": dict(n=50_000, leaves=63, bag=True),
    "small_leaves": dict(n=3000, leaves=255, noise=True, p=dict(min_data_in_leaf=2)),
    "leaves_300": dict(n=100_000, leaves=300, noise=True),
}


def _learners(lgb, c, **more):
    rng = np.random.default_rng(17)
    n, k = c["n"], c.get("k", 1)
    X = rng.standard_normal((n, 10)).astype(np.float32)
    z = X[:, 0] + X[:, 1] * X[:, 2]
    y = (rng.random(n) < (0.5 if c.get("noise") else 1 / (1 + np.exp(-z)))).astype(np.float32)
    params = {"objective": "binary", "num_leaves": c["leaves"], "num_threads": 4, "seed": 3, "use_quantized_grad": True,
              "num_grad_quant_bins": 4, "stochastic_rounding": True, "quant_train_renew_leaf": True, **c.get("p", {}), **more}
    ds = binned_dataset(lgb, X, y, params)
    return y, [lgb.Learner(ds, dict(params, persistent_grow=p), num_tree_slots=k) for p in (False, True)]


def _grads(y, k, it):
    rng = np.random.default_rng(40 + it)
    g = (0.5 - y + 0.3 * rng.standard_normal((k, len(y)))).astype(np.float32).ravel()
    h = (0.1 + 0.2 * rng.random(k * len(y))).astype(np.float32)
    # many binary orders: their FP64 sums are rounded, so another order gives other bits
    small = rng.random(len(g)) < 0.3
    g[small] = np.ldexp(g[small], -rng.integers(20, 45, int(small.sum())))
    h[::3] = np.ldexp(h[::3], -rng.integers(20, 45, len(h[::3])))
    return g, h


@pytest.mark.parametrize("case", sorted(CASES))
def test_renewed_leaves_are_those_of_growth_by_split(lgb, case):
    c = CASES[case]
    k = c.get("k", 1)
    y, (rounds, steps) = _learners(lgb, c)
    if c.get("bag"):
        used = np.sort(np.random.default_rng(1).choice(c["n"], c["n"] // 2, replace=False)).astype(np.uint32)
        rounds.set_bagging(used)
        steps.set_bagging(used)
    for it in range(3):
        g, h = _grads(y, k, it)
        for slot, (a, b) in enumerate(zip(rounds.train(g, h), steps.train(g, h))):
            assert np.array_equal(a["split_feature"], b["split_feature"])
            assert np.array_equal(a["leaf_value"], b["leaf_value"])
            nl = int(a["num_leaves"])
            for u, w in zip(rounds.partition(slot, nl), steps.partition(slot, nl)):
                assert np.array_equal(u, w)


def test_a_bag_in_no_order_keeps_every_row(lgb):
    """Rows in no order cannot be put back by rank: the leaves keep their pieces, and each row once."""
    c = CASES["plain"]
    y, (rounds, steps) = _learners(lgb, c, use_quantized_grad=False)
    used = np.random.default_rng(2).permutation(c["n"])[:c["n"] // 2].astype(np.uint32)
    rounds.set_bagging(used)
    steps.set_bagging(used)
    g, h = _grads(y, 1, 0)
    a, b = rounds.train(g, h)[0], steps.train(g, h)[0]
    assert np.array_equal(a["split_feature"], b["split_feature"])
    for u, w in zip(rounds.partition(0, int(a["num_leaves"])), steps.partition(0, int(a["num_leaves"]))):
        assert np.array_equal(u, w)
