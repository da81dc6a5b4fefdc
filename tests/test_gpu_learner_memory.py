"""Device memory of a learner: what a form of growth needs comes first, and the
pools of the explored nodes shrink to what is left, which changes no tree."""
import numpy as np
import pytest

from conftest import binned_dataset

pytestmark = pytest.mark.gpu

N, F, LEAVES = 2000, 2000, 255


@pytest.fixture(scope="module")
def wide(lgb):
    rng = np.random.default_rng(1)
    X = rng.standard_normal((N, F)).astype(np.float32)
    y = (X[:, 0] + X[:, 1] + rng.standard_normal(N) > 0).astype(np.float32)
    params = {"objective": "binary", "num_leaves": LEAVES, "min_data_in_leaf": 2, "hist_precision": "f64", "num_threads": 8}
    # on a grid, so that FP64 sums are exact in any order
    g = np.round((0.5 - y + 0.3 * rng.standard_normal(N)) * 1024).astype(np.float32) / 1024
    h = np.round((0.1 + 0.2 * rng.random(N)) * 1024).astype(np.float32) / 1024
    return binned_dataset(lgb, X, y, params), params, g, h


def _used(torch):
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_pools_shrink_to_the_memory_left(lgb, wide):
    torch = pytest.importorskip("torch")
    ds, params, g, h = wide
    learner = lgb.Learner(ds, params)
    want = learner.train(g, h)[0]
    before = _used(torch)
    del learner
    torch.cuda.empty_cache()
    took = before - _used(torch)  # with full pools
    bins = int(ds.binned()["num_bin"].sum())
    least = LEAVES * (bins - F) * 16  # one histogram a leaf
    assert took > 2 * least
    free, _ = torch.cuda.mem_get_info()
    # room for the histograms of the finished tree and a little more, not for the pools
    hold = torch.empty(free - least - (160 << 20), dtype=torch.uint8, device="cuda")
    learner = lgb.Learner(ds, params)
    got = learner.train(g, h)[0]
    del learner, hold
    torch.cuda.empty_cache()
    for name in ("num_leaves", "split_feature", "threshold_in_bin", "leaf_count", "leaf_value"):
        assert np.array_equal(got[name], want[name]), name


def test_data_parallel_growth_keeps_no_pools(lgb, wide):
    torch = pytest.importorskip("torch")
    ds, params, g, h = wide
    start = _used(torch)
    steps = lgb.Learner(ds, dict(params, persistent_grow=True))
    one = _used(torch) - start
    learner = lgb.Learner(ds, params)
    learner.set_data_parallel(0, N, lambda ptr, count, dtype, op: None)
    assert _used(torch) - start <= 2 * one + (32 << 20)
    a, b = learner.train(g, h)[0], steps.train(g, h)[0]
    assert np.array_equal(a["split_feature"], b["split_feature"])
    assert np.array_equal(a["leaf_count"], b["leaf_count"])
