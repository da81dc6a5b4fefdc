"""Batched prediction (lgbm_b200_predict) over every form its launch chooses:
few rows (the warps of a CTA share the trees) and many, rows staged or read
from global memory, trees staged or not, the compact node layout and the wide
one, against a plain FP64 walk of the same trees. The leaf values are added in
model order in both, so the scores are equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rows, columns, trees, leaves, trees per iteration, largest feature index (-1: the last column)
CASES = [
    (1, 5, 7, 31, 1, -1), (31, 28, 100, 31, 1, -1), (33, 28, 100, 31, 3, -1), (100, 136, 70, 255, 1, -1),
    (700, 1, 3, 2, 1, -1), (9471, 12, 20, 63, 1, -1), (9473, 13, 21, 63, 3, -1), (20001, 30, 9, 127, 1, -1),
    (40003, 223, 6, 255, 1, -1), (76001, 28, 10, 63, 2, -1),
    (50, 700, 10, 31, 1, -1), (12000, 700, 5, 31, 1, -1),      # fewer rows a CTA fit
    (40, 1500, 10, 31, 1, -1), (12000, 1500, 5, 31, 2, -1),    # rows read from global memory
    (90, 10, 5, 6000, 1, -1), (30000, 10, 5, 9000, 1, -1),     # trees read from global memory
    (300, 6, 4, 33000, 1, -1), (200, 40, 6, 31, 1, 9000),      # the wide layout
    (200, 8, 6, 31, 1, 20), (50, 4, 5, 1, 1, -1),              # features past the row; constant trees
]


def _forest(rng, ncol, trees, leaves, max_feature):
    out = []
    grid = np.concatenate([np.float64(np.float32(rng.standard_normal(40))), rng.standard_normal(40), [0.0, -0.0, 1e-36, 1e300]])
    for _ in range(trees):
        nn = leaves - 1
        left, right, parent = np.zeros(nn, np.int32), np.zeros(nn, np.int32), np.full(leaves, -1)
        for node in range(nn):
            leaf = int(rng.integers(0, node + 1))
            up = parent[leaf]
            if up >= 0:
                (left if left[up] == ~leaf else right)[up] = node
            left[node], right[node] = ~leaf, ~(node + 1)
            parent[leaf] = parent[node + 1] = node
        cat = rng.random(nn) < 0.1
        nc = int(cat.sum())
        thr = rng.choice(grid, nn)
        thr[cat] = np.arange(nc)
        dt = (2 * rng.integers(0, 2, nn) + 4 * rng.integers(0, 3, nn)).astype(np.int8)
        dt[cat] = 1
        z = np.zeros(nn)
        out.append({
            "num_leaves": leaves, "num_cat": nc, "left_child": left, "right_child": right,
            "leaf_parent": parent.astype(np.int32), "leaf_depth": np.zeros(leaves, np.int32),
            "split_feature": rng.integers(0, (max_feature if max_feature >= 0 else ncol - 1) + 1, nn).astype(np.int32),
            "split_feature_inner": z.astype(np.int32), "split_gain": z.astype(np.float32),
            "threshold_in_bin": z.astype(np.uint32), "threshold": thr, "decision_type": dt,
            "leaf_value": rng.standard_normal(leaves), "leaf_weight": np.ones(leaves),
            "leaf_count": np.ones(leaves, np.int32), "internal_value": z, "internal_weight": z,
            "internal_count": z.astype(np.int32), "cat_boundaries": 2 * np.arange(nc + 1, dtype=np.int32),
            "cat_threshold": rng.integers(0, 1 << 32, 2 * nc, dtype=np.uint64).astype(np.uint32),
            "cat_boundaries_inner": np.zeros(nc + 1, np.int32), "cat_threshold_inner": np.zeros(0, np.uint32)})
    return out


def _walk(t, X):
    """Leaf of every row (predict.rs:77-111) on values of which |v| <= 1e-35 counts as zero."""
    node = np.zeros(len(X), np.int64) if t["num_leaves"] > 1 else np.full(len(X), -1)
    tiny = np.float64(np.float32(1e-35))
    while (node >= 0).any():
        rows = np.nonzero(node >= 0)[0]
        n = node[rows]
        f = t["split_feature"][n]
        v = np.where(f < X.shape[1], X[rows, np.minimum(f, X.shape[1] - 1)].astype(np.float64), 0.0)
        v = np.where(np.abs(v) <= tiny, 0.0, v)
        dt, thr = t["decision_type"][n], t["threshold"][n]
        mt = (dt >> 2) & 3
        nan = np.isnan(v)
        w = np.where(nan & (mt != 2), 0.0, v)
        default = ((mt == 1) & (np.abs(w) <= tiny)) | ((mt == 2) & nan)
        left = np.where(default, (dt & 2) != 0, w <= thr)
        cat = (dt & 1) != 0
        if cat.any():
            c = np.where(nan | ~np.isfinite(v), -1, np.clip(v, -2, 1e6)).astype(np.int64)
            ci = np.where(cat, thr, 0).astype(np.int64)
            ok = (c >= 0) & (c < 64)
            word = t["cat_threshold"][2 * ci + np.where(ok, c // 32, 0)]
            left = np.where(cat, ok & ((word >> (np.where(ok, c, 0) % 32)) & 1 == 1), left)
        node[rows] = np.where(left, t["left_child"][n], t["right_child"][n])
    return ~node


@pytest.mark.parametrize("where", ["host", "device"])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_predict_equals_plain_walk(lgb, case, where):
    import torch

    rows, ncol, trees, leaves, k, max_feature = CASES[case]
    rng = np.random.default_rng(100 + case)
    model = _forest(rng, ncol, trees * k, leaves, max_feature)
    X = rng.standard_normal((rows, ncol)).astype(np.float32)
    X[rng.random(X.shape) < 0.1] = 0.0
    X[rng.random(X.shape) < 0.1] = np.nan
    X[rng.random(X.shape) < 0.05] = np.float32(1e-36)
    whole = rng.random(X.shape) < 0.2
    X[whole] = rng.integers(0, 70, int(whole.sum()))
    want = np.zeros((rows, k))
    for i, t in enumerate(model):
        want[:, i % k] += t["leaf_value"][_walk(t, X)]
    params = {"objective": "multiclass", "num_class": k} if k > 1 else {"objective": "regression"}
    bst = lgb.Booster(params)
    bst.trees = model
    if where == "host":
        got = bst.predict(X, raw_score=True).reshape(rows, k)
    else:
        # one float past a 16-byte boundary, so that the row loads cannot be vectors
        from lgbm_b200 import _lib as L

        buf = torch.zeros(rows * ncol + 1, dtype=torch.float32, device="cuda")
        buf[1:] = torch.from_numpy(X.ravel()).cuda()
        out = torch.empty(rows * k, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        L.check(L.lib().lgbm_b200_predict(bst._forest_handle(), buf.data_ptr() + 4, rows, ncol, out.data_ptr(), L.DEVICE))
        got = out.cpu().numpy().reshape(rows, k)
    assert np.array_equal(got, want)
