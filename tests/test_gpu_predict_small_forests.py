"""Prediction under forests of few or small trees, which a thread a row walks
one tree after the other, and on either side of the rule that decides it: equal
to a plain FP64 walk bit for bit (tests/test_gpu_predict_layouts.py). Trees of
different size share a forest."""
import numpy as np
import pytest

from test_gpu_predict_layouts import _forest, _walk

pytestmark = pytest.mark.gpu

# rows, columns, trees per class, leaves (taken in turn), classes, largest feature index (-1: the last column)
CASES = [
    (1, 3, 1, [7], 1, -1), (40_001, 28, 1, [31], 1, -1), (40_000, 5, 1, [2], 1, -1), (30_001, 223, 1, [63], 1, -1),
    (30_000, 224, 1, [63], 1, -1), (40_001, 28, 1, [31, 1, 200], 3, -1), (40_001, 4, 10, [2], 1, -1),
    (40_001, 4, 100, [1], 1, -1), (2000, 12, 1, [15, 3], 1000, -1), (40_001, 12, 2, [15, 1, 255], 2, -1),
    (40_001, 12, 20, [4, 1, 9], 1, -1), (30_000, 10, 20, [9000, 3], 1, -1), (40_001, 8, 1, [31], 1, 20),
    (500, 40, 3, [33_000, 5], 1, -1), (500, 300, 3, [31, 7], 2, 9000), (0, 5, 3, [7], 1, -1),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_small_forests_equal_plain_walk(lgb, case):
    import torch
    from lgbm_b200 import _lib as L

    rows, ncol, trees, leaves, k, max_feature = CASES[case]
    rng = np.random.default_rng(200 + case)
    kinds = [_forest(rng, ncol, 2, nl, max_feature) for nl in leaves]
    model = [kinds[i % len(kinds)][(i // len(kinds)) % 2] for i in range(trees * k)]
    X = rng.standard_normal((rows, ncol)).astype(np.float32)
    X[rng.random(X.shape) < 0.1] = 0.0
    X[rng.random(X.shape) < 0.1] = np.nan
    X[rng.random(X.shape) < 0.05] = np.float32(-1e-36)
    whole = rng.random(X.shape) < 0.2
    X[whole] = rng.integers(0, 70, int(whole.sum()))
    leaf_of = {id(t): t["leaf_value"][_walk(t, X)] for kind in kinds for t in kind}
    want = np.zeros((rows, k))
    for i, t in enumerate(model):
        want[:, i % k] += leaf_of[id(t)]
    bst = lgb.Booster({"objective": "multiclass", "num_class": k} if k > 1 else {"objective": "regression"})
    bst.trees = model
    for shift in (0, 1):  # a float past a 16-byte boundary, so that the row loads cannot be vectors
        buf = torch.zeros(rows * ncol + 1, dtype=torch.float32, device="cuda")
        buf[shift:shift + rows * ncol] = torch.from_numpy(X.ravel()).cuda()
        out = torch.empty(max(1, rows * k), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        L.check(L.lib().lgbm_b200_predict(bst._forest_handle(), buf.data_ptr() + 4 * shift, rows, ncol, out.data_ptr(), L.DEVICE))
        assert np.array_equal(out.cpu().numpy()[:rows * k].reshape(rows, k), want)
