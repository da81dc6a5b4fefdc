"""Lambdarank gradients of queries of a few rows, which lane groups share a
warp for, against the oracle: unnormalised bit for bit, normalised within an
ulp (CUDA's log2), as the larger queries' beside them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ulps(a, b):
    return np.abs(a.view(np.int32).astype(np.int64) - b.view(np.int32).astype(np.int64))


GROUPS = {
    "one_row": [1],
    "one_query": [5],
    "eight_and_nine": [8, 9, 8, 9, 7],
    "a_cta_and_one": [3] * 17,  # 16 queries a CTA
    "empty_between": [0, 4, 0, 0, 8, 2, 0],
    "only_large": [20, 300, 9],
    "every_size": list(range(13)) * 40,
}


@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("trunc", [1, 3, 30])
@pytest.mark.parametrize("name", sorted(GROUPS))
def test_small_queries(lgb, orc, name, trunc, norm):
    group = np.array(GROUPS[name], np.int32)
    rng = np.random.default_rng(len(group) + trunc)
    rng.shuffle(group)
    n = int(group.sum())
    label = rng.integers(0, 5, n).astype(np.float32)
    score = np.round(rng.standard_normal(n), 1)  # ties: the stable order decides
    score[rng.random(n) < 0.1] = -np.inf  # the minimum score: its pairs are skipped
    score[rng.random(n) < 0.1] = -0.0
    params = {"objective": "lambdarank", "lambdarank_norm": norm, "lambdarank_truncation_level": trunc}
    g, h = lgb.gradients(params, label, score, group=group)
    og, oh = orc.gradients(lgb.resolve_params(params), label, score, group)
    if norm:
        assert _ulps(g, og).max() <= 1 and _ulps(h, oh).max() <= 1
    else:
        assert np.array_equal(g, og) and np.array_equal(h, oh)


def test_a_ranking_booster_of_small_queries(lgb, orc):
    """The interleaved gradients of the device-resident booster."""
    rng = np.random.default_rng(5)
    group = rng.integers(1, 12, 800).astype(np.int32)
    n = int(group.sum())
    X = rng.standard_normal((n, 6)).astype(np.float32)
    y = np.clip(np.round(X[:, 0] + 0.5 * rng.standard_normal(n) + 1), 0, 4).astype(np.float32)
    params = {"objective": "lambdarank", "num_leaves": 15, "min_data_in_leaf": 5, "lambdarank_norm": False}
    ds = lgb.Dataset(X, y, group=group, params=params)
    bst = lgb.train(params, ds, num_boost_round=3)
    om = orc.train(lgb.resolve_params(params), ds.binned(), y, 3, group=group)
    for a, o in zip(bst.trees, om.trees):
        assert np.array_equal(a["split_feature"], o["split_feature"])
        assert np.array_equal(a["leaf_count"], o["leaf_count"])
