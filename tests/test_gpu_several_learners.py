"""Learners of different shape alive in one process.

The shared-memory limit of a kernel belongs to the device, not to a learner:
creating a learner must not refuse the launches of those created before it,
whatever their leaves and feature kinds."""
import numpy as np
import pytest

from conftest import binned_dataset

pytestmark = pytest.mark.gpu

FIELDS = ("num_leaves", "split_feature", "threshold_in_bin", "decision_type", "left_child", "right_child", "leaf_count",
          "cat_threshold")


def _data(n, cats):
    rng = np.random.default_rng(11)
    X = rng.standard_normal((n, 8)).astype(np.float32)
    for j in range(cats):
        X[:, 7 - j] = rng.integers(0, 30, n)
    y = (X[:, 0] + X[:, 1] * X[:, 2] + 0.5 * rng.standard_normal(n) > 0).astype(np.float32)
    return X, y


def _params(form, leaves, graph):
    p = {"objective": "binary", "num_leaves": leaves, "min_data_in_leaf": 2, "num_threads": 4, "seed": 5,
         "use_cuda_graph": graph}
    if form == "quantized":
        p.update(use_quantized_grad=True, num_grad_quant_bins=4, stochastic_rounding=True, quant_train_renew_leaf=True)
    else:
        p["hist_precision"] = form
    return p


def _grads(y, it):
    # on a grid, so that FP64 sums are exact in any order
    rng = np.random.default_rng(100 + it)
    g = np.round((0.5 - y + 0.2 * rng.standard_normal(len(y))) * 1024).astype(np.float32) / 1024
    h = np.round((0.1 + 0.2 * rng.random(len(y))) * 1024).astype(np.float32) / 1024
    return g, h


def _same(a, b):
    for name in FIELDS:
        assert np.array_equal(a[name], b[name]), name
    np.testing.assert_allclose(a["leaf_value"], b["leaf_value"], rtol=1e-9, atol=1e-12)


# the first learner, then the smaller one created after it: (leaves, categorical columns)
PAIRS = {"cats_then_none": ((255, 2), (31, 0)), "leaves": ((255, 0), (31, 0)), "many_leaves": ((4000, 0), (15, 0))}


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("form", ["quantized", "f64", "f32c"])
@pytest.mark.parametrize("pair", sorted(PAIRS))
def test_a_smaller_learner_leaves_the_larger_one_working(lgb, pair, form, graph):
    made = []
    for leaves, cats in PAIRS[pair]:
        X, y = _data(20_000, cats)
        p = _params(form, leaves, graph)
        ds = binned_dataset(lgb, X, y, p, categorical=list(range(8 - cats, 8)))
        made.append((ds, p, y))
    alone = []
    for ds, p, y in made:
        learner = lgb.Learner(ds, p)
        alone.append([learner.train(*_grads(y, it))[0] for it in range(3)])
        del learner
    both = [lgb.Learner(ds, p) for ds, p, _ in made]  # created before either is trained
    for it in range(3):
        for learner, (_, _, y), want in zip(both, made, alone):
            _same(learner.train(*_grads(y, it))[0], want[it])


def test_boosters_of_different_size_take_turns(lgb):
    X, y = _data(20_000, 2)
    big = _params("quantized", 255, True)
    small = _params("quantized", 31, True)
    alone = [lgb.train(p, lgb.Dataset(X[:, :f], y, params=p, categorical_feature=cats), num_boost_round=3).trees
             for p, f, cats in ((big, 8, [6, 7]), (small, 6, None))]
    both = [lgb.Booster(p, lgb.Dataset(X[:, :f], y, params=p, categorical_feature=cats))
            for p, f, cats in ((big, 8, [6, 7]), (small, 6, None))]
    for it in range(3):
        for bst, want in zip(both, alone):
            bst.update()
            _same(bst.trees[it], want[it])
