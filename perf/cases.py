"""The work that is timed: what a program that uses this framework has it do, through the public entry points.

A case is one call sequence of a user's program at one size:

update    one boosting iteration of the device-resident booster (`Booster.update`), with the new trees and
          the updated scores as its outputs
dropin    one iteration of a host program that keeps its scores in its own memory and uses the learner as a
          drop-in: gradients, tree, score update, all on host buffers
predict   raw scores of a batch of rows under a trained forest, rows in host or in device memory
metric    an evaluation metric of host scores

Each iteration of an `update` or `dropin` state continues the boosting of that state.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lightgbm-rust_b200"))

import lgbm_b200 as lgb  # noqa: E402
from lgbm_b200 import _lib  # noqa: E402

TREE_FIELDS = ("split_feature", "threshold_in_bin", "split_gain", "left_child", "right_child", "leaf_value",
               "leaf_weight", "leaf_count", "internal_value", "internal_count")


def listed():
    return [
        # a small table and small trees: what an iteration costs when the rows hardly matter (the 20,000-row
        # configuration, with its held-out rows), in the default FP64 form
        {"name": "update_binary_20k_f64", "kind": "update", "objective": "binary", "rows": 20000, "valid": 5000,
         "features": 28, "leaves": 31, "form": "f64"},
        # an ordinary table of odd size with full-size trees and quantized gradients
        {"name": "update_binary_500k_quant", "kind": "update", "objective": "binary", "rows": 500009, "valid": 0,
         "features": 28, "leaves": 255, "form": "quantized"},
        # the headline: 10M rows + 1M held-out x 28 features, 255 leaves, quantized gradients
        {"name": "update_binary_10m_quant", "kind": "update", "objective": "binary", "rows": 10000000,
         "valid": 1000000, "features": 28, "leaves": 255, "form": "quantized"},
        # a large table in the default FP64 form, features past one group of 32
        {"name": "update_binary_2m_f64", "kind": "update", "objective": "binary", "rows": 2000000, "valid": 0,
         "features": 37, "leaves": 255, "form": "f64"},
        # regression on 100 columns with missing values, bagging and column sampling (re-bagged each iteration)
        {"name": "update_l2_1m_f64", "kind": "update", "objective": "regression", "rows": 1000000, "valid": 0,
         "features": 100, "leaves": 255, "form": "f64"},
        # ten classes, 200 columns of which 20 are categorical: ten trees an iteration
        {"name": "update_multiclass_200k", "kind": "update", "objective": "multiclass", "rows": 200000, "valid": 0,
         "features": 200, "leaves": 127, "form": "quantized"},
        # ranking: queries of geometric sizes (about 40 rows each) x 136 columns
        {"name": "update_rank_800k_quant", "kind": "update", "objective": "lambdarank", "rows": 800000, "valid": 0,
         "features": 136, "leaves": 255, "form": "quantized"},
        # the learner as a drop-in behind a host program: gradients, tree and score update on host buffers
        {"name": "dropin_binary_1m_f32c", "kind": "dropin", "objective": "binary", "rows": 1000000, "features": 28,
         "leaves": 63, "form": "f32c"},
        # serving: a few rows under a model of 100 trees
        {"name": "predict_host_100", "kind": "predict", "rows": 100, "features": 28, "trees": 100, "leaves": 31,
         "device_rows": False, "nan": False},
        # scoring a table from host memory, missing values among the rows
        {"name": "predict_host_300k", "kind": "predict", "rows": 300007, "features": 100, "trees": 200,
         "leaves": 255, "device_rows": False, "nan": True},
        # batch scoring of device rows under the 300-tree ranking model
        {"name": "predict_device_2m", "kind": "predict", "rows": 2000000, "features": 136, "trees": 300,
         "leaves": 255, "device_rows": True, "nan": False},
        # the held-out AUC of an iteration
        {"name": "metric_auc_1m", "kind": "metric", "metric": "auc", "rows": 1000000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["update"] * 5 + ["dropin", "predict", "predict", "metric"])
    if kind == "metric":
        return {"kind": kind, "metric": rng.choice(["auc", "binary_logloss", "rmse"]), "rows": _log_int(rng, 1000, 2e6)}
    if kind == "predict":
        features = rng.randint(4, 136)
        return {"kind": kind, "rows": _log_int(rng, 1, 1e6), "features": features, "trees": rng.randint(10, 300),
                "leaves": _log_int(rng, 7, 255), "device_rows": rng.random() < 0.5, "nan": rng.random() < 0.5}
    objective = "binary"
    if kind == "update":
        objective = rng.choice(["binary", "binary", "regression", "multiclass", "lambdarank"])
    features = {"binary": rng.randint(5, 60), "regression": rng.randint(20, 110), "multiclass": rng.randint(30, 200),
                "lambdarank": rng.randint(20, 136)}[objective]
    most = min(3e6, (3e7 if objective == "multiclass" else 8e7) / features)
    case = {"kind": kind, "objective": objective, "rows": _log_int(rng, 3000, most), "features": features,
            "leaves": _log_int(rng, 15, 255), "form": rng.choice(["f64", "quantized", "quantized", "f32c"])}
    if kind == "update":
        case["valid"] = rng.choice([0, case["rows"] // 10])
    return case


# ---- inputs --------------------------------------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 2654435761 % (1 << 62) + 12345)


def _columns(case, rows, gen):
    """Feature columns of the objective's kind: (float32 [rows x features] on the GPU, categorical columns)."""
    nf, objective = case["features"], case["objective"]
    X = torch.randn(rows, nf, generator=gen, device="cuda")
    cats = []
    if objective == "binary":  # a quarter of the columns are products and ratios (heavy tails)
        q = nf // 4
        for k in range(q):
            a, b = X[:, k], X[:, (k + 1) % (nf - q)]
            X[:, nf - q + k] = a * b if k % 2 == 0 else a / (b.abs() + 0.1)
    elif objective == "regression":  # normal, lognormal and small whole numbers, 5% missing
        a, b = nf * 6 // 10, nf * 9 // 10
        X[:, a:b] = X[:, a:b].exp()
        X[:, b:] = torch.randint(0, 16, (rows, nf - b), generator=gen, device="cuda").float()
    elif objective == "multiclass":  # a tenth of the columns categorical, Zipf over 50 categories
        nc = nf // 10
        p = 1.0 / torch.arange(1, 51, device="cuda") ** 1.2
        for j in range(nf - nc, nf):
            X[:, j] = torch.multinomial(p, rows, replacement=True, generator=gen).float()
            cats.append(j)
    else:  # half uniform, a fifth of the values zero
        X[:, nf // 2:] = torch.rand(rows, nf - nf // 2, generator=gen, device="cuda")
        X[torch.rand(rows, nf, generator=gen, device="cuda") < 0.2] = 0.0
    return X, cats


def _labels(case, X, gen):
    rows, nf = X.shape
    objective = case["objective"]
    noise = torch.randn(rows, generator=gen, device="cuda")
    if objective == "binary":
        z = X[:, 0] + X[:, 1] * X[:, 2] - 0.5 * X[:, 3] ** 2 + 0.3 * noise
        return (torch.rand(rows, generator=gen, device="cuda") < torch.sigmoid(z)).float(), None
    if objective == "regression":
        y = torch.sin(X[:, 0]) + 0.1 * noise
        for j in range(min(10, nf)):
            y += (0.3 * j - 1.2) * (X[:, (7 * j) % nf] > 0.2 * j - 0.8)
        return y, None
    if objective == "multiclass":
        w = torch.randn(nf - nf // 10, 10, generator=gen, device="cuda") / math.sqrt(nf)
        u = torch.rand(rows, 10, generator=gen, device="cuda")
        return (X[:, : nf - nf // 10] @ w - torch.log(-torch.log(u))).argmax(1).float(), None
    w = torch.randn(nf, generator=gen, device="cuda") / math.sqrt(nf)
    s = X @ w + 0.5 * noise
    cuts = torch.quantile(s[:100000], torch.tensor([0.5, 0.75, 0.9, 0.97], device="cuda"))
    group = []
    sizes = np.random.default_rng(gen.initial_seed()).geometric(1.0 / 40.0, rows).clip(1, 1000)
    ends = np.cumsum(sizes)
    group = sizes[: int(np.searchsorted(ends, rows))].tolist()
    group.append(rows - sum(group))
    return torch.searchsorted(cuts, s).float(), [g for g in group if g > 0]


def _params(case, cats):
    p = {"objective": case["objective"], "num_leaves": case["leaves"], "learning_rate": 0.1, "device_binning": True}
    if case["form"] == "quantized":
        p.update(use_quantized_grad=True, num_grad_quant_bins=4, stochastic_rounding=True, quant_train_renew_leaf=True)
    else:
        p["hist_precision"] = case["form"]
    if case["objective"] == "regression":
        p.update(bagging_fraction=0.8, bagging_freq=1, feature_fraction=0.8, learning_rate=0.05)
    if case["objective"] == "multiclass":
        p.update(num_class=10, categorical_feature=cats, max_cat_to_onehot=4)
    return p


def _dataset(case, rows, gen, reference=None):
    X, cats = _columns(case, rows, gen)
    y, group = _labels(case, X, gen)
    if case["objective"] == "regression":
        X[torch.rand(X.shape, generator=gen, device="cuda") < 0.05] = float("nan")
    params = _params(case, cats)
    ds = lgb.Dataset(X.cpu().numpy(), y.cpu().numpy(), group=group, categorical_feature=cats, params=params,
                     reference=reference)
    return ds, params


def _forest(case, seed):
    """A trained model's trees: leaves split one at a time at random, thresholds over the columns' range."""
    rng = np.random.default_rng(seed)
    trees = []
    nl, nf = case["leaves"], case["features"]
    for _ in range(case["trees"]):
        nn = nl - 1
        left, right = np.zeros(nn, np.int32), np.zeros(nn, np.int32)
        parent, depth = np.full(nl, -1, np.int32), np.zeros(nl, np.int32)
        at = rng.random(nn)
        for node in range(nn):
            leaf = int(at[node] * (node + 1))
            up = parent[leaf]
            if up >= 0:
                (left if left[up] == ~leaf else right)[up] = node
            left[node], right[node] = ~leaf, ~(node + 1)
            parent[leaf] = parent[node + 1] = node
            depth[leaf] = depth[node + 1] = depth[leaf] + 1
        trees.append({
            "num_leaves": nl, "num_cat": 0, "left_child": left, "right_child": right, "leaf_parent": parent,
            "leaf_depth": depth, "split_feature": rng.integers(0, nf, nn).astype(np.int32),
            "split_feature_inner": np.zeros(nn, np.int32), "split_gain": np.ones(nn, np.float32),
            "threshold_in_bin": np.zeros(nn, np.uint32), "threshold": rng.standard_normal(nn),
            "decision_type": ((2 << 2 if case["nan"] else 0) | 2 * rng.integers(0, 2, nn)).astype(np.int8),
            "leaf_value": 0.1 * rng.standard_normal(nl), "leaf_weight": np.ones(nl), "leaf_count": np.ones(nl, np.int32),
            "internal_value": np.zeros(nn), "internal_weight": np.zeros(nn), "internal_count": np.ones(nn, np.int32),
            "cat_boundaries": np.zeros(1, np.int32), "cat_threshold": np.zeros(0, np.uint32),
            "cat_boundaries_inner": np.zeros(1, np.int32), "cat_threshold_inner": np.zeros(0, np.uint32)})
    return trees


class _Forest:
    """A forest handle of the C interface over the trees' arrays."""

    def __init__(self, trees):
        keep, views = [], (_lib.TreeView * len(trees))()
        for v, t in zip(views, trees):
            v.num_leaves, v.num_cat = t["num_leaves"], t["num_cat"]
            for name, kind in _lib.TreeView._fields_:
                if name in t and name not in ("num_leaves", "num_cat"):
                    a = np.ascontiguousarray(t[name]) if len(t[name]) else np.zeros(1, t[name].dtype)
                    keep.append(a)
                    setattr(v, name, ctypes.cast(a.ctypes.data, kind))
        self.handle = ctypes.c_void_p()
        _lib.check(_lib.lib().lgbm_b200_forest_create(views, len(trees), 1, 0, ctypes.byref(self.handle)))

    def __del__(self):
        if self.handle:
            _lib.lib().lgbm_b200_forest_destroy(self.handle)
            self.handle = None


def _rows(case, seed):
    gen = _generator(seed)
    X = torch.randn(case["rows"], case["features"], generator=gen, device="cuda")
    if case["nan"]:
        X[torch.rand(X.shape, generator=gen, device="cuda") < 0.05] = float("nan")
    return X


def _scored(case, seed):
    gen = _generator(seed)
    y = torch.rand(case["rows"], generator=gen, device="cuda") < 0.4
    s = (y.double() + 1.3 * torch.randn(case["rows"], generator=gen, device="cuda", dtype=torch.float64))
    s = torch.round(s * 4096) / 4096  # some equal scores, as rows that share their leaves have
    return y.float().cpu().numpy(), s.cpu().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "predict":
        trees, X = _forest(case, seed), _rows(case, seed)
        if case["device_rows"]:
            out = torch.empty(case["rows"], dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            return {"case": case, "forest": _Forest(trees), "X": X, "out": out}
        bst = lgb.Booster({"objective": "regression"})
        bst.trees = trees
        bst.predict(X[:1].cpu().numpy(), raw_score=True)  # the model is on the device before it serves
        return {"case": case, "bst": bst, "X": X.cpu().numpy()}
    if kind == "metric":
        label, scores = _scored(case, seed)
        return {"case": case, "label": label, "scores": scores}
    gen = _generator(seed)
    ds, params = _dataset(case, case["rows"], gen)
    if kind == "dropin":
        # a host program's buffers, page-locked as a program that passes them every iteration keeps them
        n = case["rows"]
        buf = {"scores": torch.zeros(n, dtype=torch.float64, pin_memory=True).numpy(),
               "grad": torch.empty(n, dtype=torch.float32, pin_memory=True).numpy(),
               "hess": torch.empty(n, dtype=torch.float32, pin_memory=True).numpy()}
        return {"case": case, "learner": lgb.Learner(ds, params), "objective": lgb.Objective(params, ds.label), **buf}
    valid = None
    if case["valid"]:
        valid = _dataset(case, case["valid"], gen, reference=ds)[0]
    bst = lgb.Booster(params, ds, valid)
    state = {"case": case, "bst": bst,
             "train": torch.empty(bst.num_class * bst.num_train, dtype=torch.float64, device="cuda")}
    if valid is not None:
        state["valid"] = torch.empty(bst.num_class * bst.num_valid, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return state


# ---- one pass ------------------------------------------------------------------------------------------------


def _update(state):
    bst = state["bst"]
    bst.update()
    trees = bst.trees[-bst.num_class:]
    out = {name: np.concatenate([t[name] for t in trees]) for name in TREE_FIELDS}
    for which, name in enumerate(("train", "valid")):
        if name in state:
            _lib.check(_lib.lib().lgbm_b200_booster_scores(bst._b, which, state[name].data_ptr(), _lib.DEVICE))
            out["scores_" + name] = state[name]
    return out


def _dropin(state):
    g, h = state["objective"].gradients(state["scores"], state["grad"], state["hess"])
    tree = state["learner"].train(g, h)[0]
    state["learner"].add_leaf_outputs(0, 0.1 * tree["leaf_value"], state["scores"])
    return {"grad": g, "hess": h, "scores": state["scores"], **{name: tree[name] for name in TREE_FIELDS}}


def _predict(state):
    if "bst" in state:
        return state["bst"].predict(state["X"], raw_score=True)
    X, out = state["X"], state["out"]
    _lib.check(_lib.lib().lgbm_b200_predict(state["forest"].handle, X.data_ptr(), X.shape[0], X.shape[1],
                                            out.data_ptr(), _lib.DEVICE))
    return out


def run(state):
    kind = state["case"]["kind"]
    if kind == "update":
        return _update(state)
    if kind == "dropin":
        return _dropin(state)
    if kind == "predict":
        return _predict(state)
    return lgb.metric(state["case"]["metric"], state["label"], state["scores"])


def work(case):
    """Inputs read once and outputs written once: the bins and per-row values of an iteration, the rows, trees
    and scores of a prediction. Operations: one pair of histogram sums per row and feature, a comparison per row
    and tree level, a few per scored row."""
    n = case["rows"]
    if case["kind"] == "metric":
        return {"bytes": 12 * n, "flops": n * max(1.0, math.log2(n))}
    if case["kind"] == "predict":
        return {"bytes": n * (4 * case["features"] + 8) + case["trees"] * case["leaves"] * 24,
                "flops": n * case["trees"] * math.log2(case["leaves"])}
    k = 10 if case["objective"] == "multiclass" else 1
    per_row = case["features"] + 4 + 16 * k + (16 if case["kind"] == "dropin" else 0)
    nv = case.get("valid", 0)
    return {"bytes": n * per_row + nv * (case["features"] + 16 * k), "flops": 2.0 * n * case["features"] * k}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------


def _exact_predict(case, seed):
    X = _rows(case, seed)
    total = torch.zeros(case["rows"], dtype=torch.float64, device="cuda")
    nl = case["leaves"]
    for t in _forest(case, seed):
        children = torch.tensor(np.stack([t["left_child"], t["right_child"]], 1), device="cuda").long()
        feature = torch.tensor(t["split_feature"], device="cuda").long()
        threshold = torch.tensor(t["threshold"], device="cuda")
        default_left = torch.tensor((t["decision_type"] & 2) != 0, device="cuda")
        value = torch.tensor(t["leaf_value"], device="cuda")
        for a in range(0, case["rows"], 1 << 19):
            x = X[a:a + (1 << 19)]
            node = torch.zeros(len(x), dtype=torch.long, device="cuda")
            for _ in range(int(t["leaf_depth"].max())):
                i = node.clamp(min=0)
                v = x.gather(1, feature[i][:, None])[:, 0].double()
                left = torch.where(torch.isnan(v), default_left[i], v <= threshold[i])
                child = children[i, (~left).long()]
                node = torch.where(node >= 0, child, node)
            total[a:a + (1 << 19)] += value[(-1 - node).clamp(0, nl - 1)]
    return total


def _exact_metric(case, seed):
    label, s = _scored(case, seed)
    y = label.astype(np.float64)
    if case["metric"] == "rmse":
        return float(np.sqrt(np.mean((s - y) ** 2)))
    if case["metric"] == "binary_logloss":
        return float(np.mean(np.logaddexp(0.0, np.where(y > 0, -s, s))))
    values, at = np.unique(s, return_inverse=True)
    pos = np.bincount(at, weights=y, minlength=len(values))
    neg = np.bincount(at, weights=1.0 - y, minlength=len(values))
    below = np.cumsum(neg) - neg
    return float(np.sum(pos * (below + 0.5 * neg)) / (pos.sum() * neg.sum()))


def exact(case, seed):
    if case["kind"] == "predict":
        total = _exact_predict(case, seed)
        return total if case["device_rows"] else total.cpu().numpy()
    if case["kind"] == "metric":
        return _exact_metric(case, seed)
    if case["kind"] == "dropin":  # the first pass's gradients, at scores of zero; the tree has no closed form
        gen = _generator(seed)
        X, _ = _columns(case, case["rows"], gen)
        y = _labels(case, X, gen)[0].double().cpu().numpy()
        return {"grad": 0.5 - y, "hess": np.full(case["rows"], 0.25), "scores": None,
                **{name: None for name in TREE_FIELDS}}
    return None  # an iteration's outputs follow from the splits it chose, which are whole numbers of the tree itself
