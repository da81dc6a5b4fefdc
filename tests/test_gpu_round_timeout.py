"""A partition that gave up waiting ends the tree in its own round. The status
is set by the host (LGBM_B200_FAIL_ROUND, on the path that launches the rounds
one by one): no kernel waits for anything."""
import numpy as np
import pytest

from conftest import binned_dataset

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots", [1, 2])
@pytest.mark.parametrize("fail", [0, 1, 3])
def test_growth_ends_in_the_round_that_failed(lgb, monkeypatch, fail, slots):
    rng = np.random.default_rng(0)
    n = 20_000
    X = rng.standard_normal((n, 6)).astype(np.float32)
    y = (X[:, 0] + X[:, 1] * X[:, 2] > 0).astype(np.float32)
    params = {"objective": "binary", "num_leaves": 127, "use_cuda_graph": False, "num_threads": 4}
    learner = lgb.Learner(binned_dataset(lgb, X, y, params), params, num_tree_slots=slots)
    g, h = np.tile((0.5 - y).astype(np.float32), slots), np.full(n * slots, 0.25, np.float32)
    learner.set_timing(True)
    want = learner.train(g, h)
    rounds = len(learner.step_times())
    assert rounds > 6
    monkeypatch.setenv("LGBM_B200_FAIL_ROUND", str(fail))
    with pytest.raises(lgb.LightGBMError, match="timed out"):
        learner.train(g, h)
    if slots == 1:  # other slots' trees go on
        assert len(learner.step_times()) == fail + 1
    monkeypatch.delenv("LGBM_B200_FAIL_ROUND")
    for a, b in zip(learner.train(g, h), want):  # the learner is usable afterwards
        assert np.array_equal(a["split_feature"], b["split_feature"])
        assert np.array_equal(a["leaf_count"], b["leaf_count"])
