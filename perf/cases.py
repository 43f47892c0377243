"""Workloads of the GBDT backend, each through the public entry points of ``mpsboost_gb300``.

``listed()`` names the workloads, ``draw()`` makes another one of the same ranges,
``prepare()`` builds the inputs a program holds before the call, ``run()`` makes the call
and returns what it computes, ``work()`` counts what a call cannot do without, and
``exact()`` restates a call in 64 bits with plain torch and numpy.

The kinds of workload:

* ``fit``      estimator fit from a float32 matrix in host memory: quantile binning on the
               device, boosting, trees and training predictions back.
* ``softmax``  the same for the native multiclass classifier (one tree per class and round).
* ``boost``    boosting on a dataset that is binned and resident already, as a parameter
               search or a cross-validation runs it.
* ``ovr``      one-vs-rest boosting on a resident dataset, the classes' trees side by side.
* ``forest``   independent deep trees on bootstrap samples of a resident dataset.
* ``score``    a float32 batch binned with a schema and run through a model.
* ``layer``    the node-level histogram hook a host tree builder calls per depth level.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import mpsboost_gb300 as mb
from mpsboost_gb300._lib import NODE_DTYPE

_BACKENDS: dict = {}


def _backend() -> mb.CudaBackend:
    """The process's one backend: a program makes it once."""

    if 0 not in _BACKENDS:
        _BACKENDS[0] = mb.CudaBackend(0)
    return _BACKENDS[0]


# --------------------------------------------------------------------------------------
# Cases
# --------------------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # A classroom-sized three-class fit: every launch and allocation counts.
        dict(name="softmax_2k", kind="softmax", rows=2_000, features=12, classes=3, trees=10, depth=4,
             bins=255, missing=0.0),
        # The plain regressor configuration: 100,000 x 32, 50 trees of depth 6.
        dict(name="fit_100k", kind="fit", rows=100_000, features=32, trees=50, depth=6, bins=255,
             missing=0.0, objective="squared_error", weighted=False),
        # A wide table with missing cells and an odd row count, binned and fitted once.
        dict(name="fit_1m_missing", kind="fit", rows=1_000_003, features=100, trees=10, depth=6, bins=255,
             missing=0.05, objective="binary_logistic", weighted=False),
        # The regression-at-scale configuration: weighted squared error, depth 8.
        dict(name="boost_10m", kind="boost", rows=10_000_000, features=128, trees=20, depth=8, bins=255,
             missing=0.0, low_card=0, objective="squared_error", weighted=True, leaves=0),
        # The binary-logistic configuration's shape: missing cells, low-cardinality
        # features, depth 10.
        dict(name="boost_logistic_missing", kind="boost", rows=1_000_000, features=256, trees=10, depth=10,
             bins=255, missing=0.1, low_card=56, objective="binary_logistic", weighted=False, leaves=0),
        # Leaf-wise growth on a mid-sized table with a ragged feature count.
        dict(name="boost_leafwise", kind="boost", rows=300_007, features=50, trees=10, depth=8, bins=255,
             missing=0.0, low_card=5, objective="squared_error", weighted=False, leaves=31),
        # Fine bins: u16 storage.
        dict(name="boost_1024bins", kind="boost", rows=1_000_000, features=64, trees=5, depth=8, bins=1024,
             missing=0.0, low_card=0, objective="squared_error", weighted=True, leaves=0),
        # The one-vs-rest configuration: ten classes, depth 6.
        dict(name="ovr_1m", kind="ovr", rows=1_000_000, features=64, classes=10, trees=5, depth=6, bins=255,
             missing=0.0),
        # The random-forest configuration: depth 12, sqrt(features), Poisson(1) rows.
        dict(name="forest_500k", kind="forest", rows=500_000, features=100, trees=32, depth=12, bins=255),
        # Batch scoring of fresh rows: binned on the device, then a 100-tree model.
        dict(name="score_1m", kind="score", rows=1_000_000, features=64, trees=100, depth=6, bins=255,
             missing=0.05, where="device"),
        # One small request: binned on the host, then the model.
        dict(name="score_1k", kind="score", rows=1_000, features=32, trees=50, depth=6, bins=255,
             missing=0.05, where="host"),
        # A host tree builder's level: sixteen nodes of a 200,000-row dataset.
        dict(name="layer_200k", kind="layer", rows=200_000, features=64, nodes=16, bins=255, missing=0.05),
    ]


def draw(rng) -> dict:
    """One more case: sizes spread over the listed ranges' logarithms, odd ones among them."""

    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["softmax", "fit", "fit", "boost", "boost", "boost", "ovr", "forest", "score", "layer"])
    bins = rng.choice([255, 255, 256, 127, 63])
    missing = rng.choice([0.0, 0.05, 0.1])
    if bins == 256:  # 256 bins and missing values are a u16 dataset of their own
        missing = 0.0
    if kind == "softmax":
        return dict(kind=kind, rows=logint(500, 60_000), features=rng.randint(4, 50), classes=rng.randint(3, 6),
                    trees=rng.randint(3, 10), depth=rng.randint(3, 6), bins=bins, missing=missing)
    if kind == "fit":
        return dict(kind=kind, rows=logint(1_000, 1_000_000), features=rng.randint(5, 100),
                    trees=rng.randint(5, 30), depth=rng.randint(3, 8), bins=bins, missing=missing,
                    objective=rng.choice(["squared_error", "binary_logistic"]), weighted=rng.random() < 0.3)
    if kind == "boost":
        wide = rng.random() < 0.2
        features = rng.randint(8, 200)
        leafwise = not wide and rng.random() < 0.2
        return dict(kind=kind, rows=logint(5_000, 300_000 if leafwise else 2_000_000), features=features,
                    trees=rng.randint(4, 10), depth=rng.randint(4, 10), bins=rng.choice([300, 1024, 2000]) if wide else bins,
                    missing=missing, low_card=rng.randint(0, features // 4),
                    objective=rng.choice(["squared_error", "binary_logistic"]), weighted=rng.random() < 0.5,
                    leaves=rng.randint(8, 40) if leafwise else 0)
    if kind == "ovr":
        return dict(kind=kind, rows=logint(10_000, 1_000_000), features=rng.randint(8, 64), classes=rng.randint(3, 10),
                    trees=rng.randint(2, 5), depth=rng.randint(4, 7), bins=bins, missing=missing)
    if kind == "forest":
        return dict(kind=kind, rows=logint(10_000, 500_000), features=rng.randint(16, 120), trees=rng.randint(4, 32),
                    depth=rng.randint(6, 12), bins=bins)
    if kind == "score":
        return dict(kind=kind, rows=logint(300, 1_000_000), features=rng.randint(8, 64), trees=rng.randint(10, 100),
                    depth=rng.randint(4, 8), bins=bins, missing=missing, where=rng.choice(["device", "host"]))
    return dict(kind=kind, rows=logint(5_000, 400_000), features=rng.randint(8, 64), nodes=rng.randint(1, 32),
                bins=bins, missing=missing)


# --------------------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------------------
def _device() -> str:
    return "cuda" if torch.cuda.is_available() else "cpu"


def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) * 1_000_003 + 17)
    return g


def _signal(z: torch.Tensor, g: torch.Generator, noise: float = 0.5) -> torch.Tensor:
    """Regression target of feature columns z [features, rows]: a sine, a square and random
    pairwise products, with noise (FP64)."""

    f, n = z.shape
    pairs = torch.randint(0, f, (8, 2), generator=g, device=z.device).tolist()
    y = torch.sin(z[0].double()) + 0.5 * z[f // 2].double() ** 2
    for a, b in pairs:
        y += z[a].double() * z[b].double()
    return y + noise * torch.randn(n, generator=g, device=z.device, dtype=torch.float64)


def _labels(case: dict, z: torch.Tensor, g: torch.Generator) -> torch.Tensor:
    y = _signal(z, g)
    if case.get("objective") == "binary_logistic":
        p = torch.sigmoid(0.7 * (y - y.mean()))
        return (torch.rand(p.shape, generator=g, device=p.device, dtype=torch.float64) < p).double()
    return y


def _class_labels(z: torch.Tensor, classes: int, g: torch.Generator) -> torch.Tensor:
    """argmax of random linear scores plus Gumbel noise."""

    w = torch.randn(classes, z.shape[0], generator=g, device=z.device)
    u = torch.rand(classes, z.shape[1], generator=g, device=z.device).clamp_(1e-7, 1 - 1e-7)
    y = (w @ z - torch.log(-torch.log(u))).argmax(0).double()
    y[:classes] = torch.arange(classes, device=z.device, dtype=torch.float64)  # every class occurs
    return y


def _matrix(case: dict, g: torch.Generator) -> torch.Tensor:
    """[features, rows] float32 on the device, before missing cells are cut out: normal
    features, every fourth log-normal, every fifth a whole number in [0, 1000)."""

    f, n = case["features"], case["rows"]
    z = torch.randn(f, n, generator=g, device=_device())
    z[3::4] = torch.exp(z[3::4])
    z[4::5] = torch.randint(0, 1000, z[4::5].shape, generator=g, device=z.device).float()
    return z


def _scaled(z: torch.Tensor) -> torch.Tensor:
    """The columns on a common scale, for the labels."""

    s = z.clone()
    s[3::4] /= 1.65
    s[4::5] /= 500.0
    return s


def _with_missing(case: dict, z: torch.Tensor, g: torch.Generator) -> np.ndarray:
    """Row-major float32 host matrix with the case's share of NaN cells."""

    if case["missing"]:
        z = z.masked_fill(torch.rand(z.shape, generator=g, device=z.device) < case["missing"], float("nan"))
    return z.t().contiguous().cpu().numpy()


def _bin_counts(case: dict) -> np.ndarray:
    counts = np.full(case["features"], case["bins"], np.uint32)
    low = case.get("low_card", 0)
    if low:
        counts[-low:] = 2 + np.arange(low) % 15
    return counts


def _binned(case: dict, g: torch.Generator, keep_z: bool = True):
    """A quantile-binned dataset (bins of a continuous feature are uniform) and columns z
    the labels are made from (a missing cell reads as 0)."""

    f, n = case["features"], case["rows"]
    counts = _bin_counts(case)
    wide = case["bins"] > 256
    dev = _device()
    bins = torch.empty(f, n, dtype=torch.int16 if wide else torch.uint8, device=dev)
    top = 24 if keep_z else 0  # columns the labels use
    used = sorted({int(i * f / top) for i in range(top)}) if top else []
    z = torch.empty(len(used), n, device=dev)
    missing = None
    if case.get("missing", 0.0):
        missing = torch.empty(f, n, dtype=torch.bool, device=dev)
    for i in range(f):
        b = torch.randint(0, int(counts[i]), (n,), generator=g, device=dev, dtype=bins.dtype)
        if i in used:
            u = (b.float() + 0.5) / float(counts[i])
            z[used.index(i)] = math.sqrt(2.0) * torch.erfinv(2.0 * u - 1.0)
        if missing is not None:
            m = torch.rand(n, generator=g, device=dev) < case["missing"]
            missing[i] = m
            b = b.masked_fill(m, 0)
            if i in used:
                z[used.index(i)].masked_fill_(m, 0.0)
        bins[i] = b
    host_bins = bins.cpu().numpy()
    if wide:
        host_bins = host_bins.view(np.uint16)
    offsets = np.concatenate([[0], np.cumsum(counts - 1)])[:-1].astype(np.uint64)
    bounds = np.concatenate([np.arange(1, c, dtype=np.float32) for c in counts])
    host_missing = missing.cpu().numpy() if missing is not None else np.zeros((f, n), bool)
    miss_counts = (missing.sum(1).cpu().numpy() if missing is not None else np.zeros(f)).astype(np.uint64)
    ds = mb.BinnedDataset(n, f, case["bins"], host_bins, host_missing, bounds, offsets,
                          (counts - 1).astype(np.uint32), counts, miss_counts)
    return ds, z


def _random_trees(case: dict, counts: np.ndarray, rng: np.random.Generator) -> list[np.ndarray]:
    """Complete trees of the case's depth: random features, thresholds around the middle,
    small leaves (a boosted model's shape)."""

    trees, inner = [], (1 << case["depth"]) - 1
    for _ in range(case["trees"]):
        t = np.zeros(2 * inner + 1, NODE_DTYPE)
        feats = rng.integers(0, case["features"], inner)
        t["feature_index"][:inner] = feats
        t["threshold_bin"][:inner] = np.maximum(
            0, (counts[feats] - 1) * rng.uniform(0.2, 0.8, inner) - 0.5).astype(np.uint32)
        t["left_child"][:inner] = 2 * np.arange(inner) + 1
        t["right_child"][:inner] = 2 * np.arange(inner) + 2
        t["left_child"][inner:] = t["right_child"][inner:] = 0xFFFFFFFF
        t["gain"][:inner] = 1.0
        t["default_left"] = rng.integers(0, 2, t.size)
        t["flags"][inner:] = 1
        t["leaf_value"][inner:] = rng.normal(0.0, 0.3, inner + 1)
        trees.append(t)
    return trees


def _host(t: torch.Tensor | None) -> np.ndarray | None:
    return None if t is None else t.cpu().numpy()


def _fit_inputs(case: dict, seed: int):
    """(matrix, labels, weights) of a fit or softmax case."""

    g = _generator(seed)
    z = _matrix(case, g)
    if case["kind"] == "softmax":
        y = _class_labels(_scaled(z), case["classes"], g)
    else:
        y = _labels(case, _scaled(z), g)
    w = 0.5 + torch.rand(case["rows"], generator=g, device=z.device, dtype=torch.float64) if case.get("weighted") else None
    return _with_missing(case, z, g), _host(y), _host(w)


def _boost_inputs(case: dict, seed: int):
    """(binned dataset, labels, weights) of a boost or one-vs-rest case."""

    g = _generator(seed)
    ds, z = _binned(case, g)
    y = _class_labels(z, case["classes"], g) if case["kind"] == "ovr" else _labels(case, z, g)
    w = 0.5 + torch.rand(case["rows"], generator=g, device=z.device, dtype=torch.float64) if case.get("weighted") else None
    return ds, _host(y), _host(w)


def _boost_params(case: dict) -> dict:
    p = dict(n_estimators=case["trees"], max_depth=case["depth"], learning_rate=0.1, min_samples_leaf=20,
             min_child_weight=1.0, reg_lambda=1.0, max_bins=case["bins"])
    if case["kind"] == "boost":
        p["objective"] = case["objective"]
    if case.get("leaves"):
        p.update(growth_strategy="leaf_wise", max_leaves=case["leaves"])
    return p


def _layer_inputs(case: dict, seed: int):
    g = _generator(seed)
    ds, z = _binned(case, g)
    y = _signal(z, g)
    pairs = torch.stack([y.mean() - y, torch.ones_like(y)], 1)
    node = torch.randint(0, case["nodes"], (case["rows"],), generator=g, device=y.device)
    node[: case["nodes"]] = torch.arange(case["nodes"], device=y.device)
    node = node.cpu().numpy()
    rows = [np.flatnonzero(node == k).astype(np.uint64) for k in range(case["nodes"])]
    return ds, _host(pairs), rows


def _score_inputs(case: dict, seed: int):
    """(training matrix for the schema, matrix to score, trees without bin counts' scale)."""

    g = _generator(seed)
    train = dict(case, rows=20_000)
    return _with_missing(train, _matrix(train, g), g), _with_missing(case, _matrix(case, g), g)


def _estimator(case: dict):
    common = dict(n_estimators=case["trees"], max_depth=case["depth"], max_bins=case["bins"], learning_rate=0.1)
    if case["kind"] == "softmax":
        return mb.GradientBoostingClassifier(multi_strategy="softmax", **common)
    if case["objective"] == "binary_logistic":
        return mb.GradientBoostingClassifier(**common)
    return mb.GradientBoostingRegressor(**common)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    s: dict = {"case": case}
    if kind in ("fit", "softmax"):
        s["x"], s["y"], s["w"] = _fit_inputs(case, seed)
        s["estimator"] = _estimator(case)
        return s
    b = s["backend"] = _backend()
    if kind in ("boost", "ovr"):
        s["data"], s["y"], s["w"] = _boost_inputs(case, seed)
        s["params"] = _boost_params(case)
        b.dataset(s["data"])  # resident
    elif kind == "forest":
        g = _generator(seed)
        s["data"], z = _binned(case, g)
        s["y"] = _host(_signal(z, g, noise=1.0))
        rng = np.random.default_rng(seed)
        n, f = case["rows"], case["features"]
        counts = torch.poisson(torch.ones(case["trees"], n, device=_device()), generator=g)
        counts[:, :2] = 1.0  # no empty sample
        s["counts"] = counts.clamp_(max=255.0).to(torch.uint8).cpu().numpy()
        k = max(1, math.ceil(math.sqrt(f)))
        s["subsets"] = [np.sort(rng.choice(f, k, replace=False)) for _ in range(case["trees"])]
        s["params"] = dict(max_depth=case["depth"], min_samples_leaf=5, min_child_weight=1.0, max_bins=case["bins"])
        b.dataset(s["data"])
    elif kind == "score":
        train, s["x"] = _score_inputs(case, seed)
        rng = np.random.default_rng(seed)
        s["schema"] = (mb.quantize_device(b, train, case["bins"]) if case["where"] == "device"
                       else mb.quantize_dense(train, case["bins"]))
        s["model"] = mb.RegressionModel(0.25, 0.1, _random_trees(case, s["schema"].bin_counts.astype(np.int64), rng))
    else:
        s["data"], s["pairs"], s["rows"] = _layer_inputs(case, seed)
        b.dataset(s["data"])
    return s


# --------------------------------------------------------------------------------------
# Calls
# --------------------------------------------------------------------------------------
def _nodes(trees: list[np.ndarray], case: dict) -> dict:
    """The trees' nodes one after another, with room for the largest trees of the case."""

    t = np.concatenate(trees)
    room = len(trees) * ((2 * case["leaves"] if case.get("leaves") else 2 << case["depth"]) - 1)
    out = {}
    for name in ("feature_index", "threshold_bin", "left_child", "right_child", "leaf_value", "gain",
                 "default_left", "flags"):
        out[name] = np.zeros(room, t[name].dtype)
        out[name][: t.size] = t[name]
    out["sizes"] = np.asarray([x.size for x in trees], np.int64)
    return out


def _model(m, case: dict) -> dict:
    return {"base": float(m.base_score), "predictions": m.train_predictions, "trees": _nodes(m.trees, case)}


def run(state: dict) -> dict:
    case, kind = state["case"], state["case"]["kind"]
    if kind == "fit":
        return _model(state["estimator"].fit(state["x"], state["y"], state["w"]).model_.model, case)
    if kind == "softmax":
        m = state["estimator"].fit(state["x"], state["y"]).model_
        return {"base": m.base_scores, "predictions": m.train_margins, "trees": _nodes(m.trees, case)}
    b = state["backend"]
    if kind == "boost":
        return _model(mb.train_regressor(b, state["data"], state["y"], state["w"], **state["params"]), case)
    if kind == "ovr":
        models = mb.train_ovr(b, state["data"], state["y"], case["classes"], **state["params"])
        return {"base": [float(m.base_score) for m in models], "predictions": [m.train_predictions for m in models],
                "trees": _nodes([t for m in models for t in m.trees], case)}
    if kind == "forest":
        models = mb.train_forest(b, state["data"], state["y"], row_counts=state["counts"],
                                 feature_subsets=state["subsets"], **state["params"])
        return {"base": np.asarray([m.base_score for m in models]), "trees": _nodes([m.trees[0] for m in models], case)}
    if kind == "score":
        data = state["schema"].transform(state["x"])
        return {"predictions": state["model"].predict(b, data)}
    hists = b.layer_histograms(state["data"], state["pairs"], state["rows"])
    h = np.concatenate([f for node in hists for f in node])
    return {"count": h["count"].astype(np.int64), "gradient": h["gradient_sum"], "hessian": h["hessian_sum"]}


def work(case: dict) -> dict:
    """Bytes and operations of one call: a tree reads every bin of its rows once and its
    rows' label, weight and prediction, and writes the prediction; a cell adds a count, a
    gradient and a hessian."""

    n, f, kind = case["rows"], case["features"], case["kind"]
    cells = n * f
    if kind == "layer":
        return {"bytes": cells + n * (8 + 16) + case["nodes"] * f * case["bins"] * 24, "flops": 3 * cells}
    if kind == "score":
        return {"bytes": 4 * cells + n * (f + 8), "flops": n * case["trees"] * (case["depth"] + 2)}
    trees = case["trees"] * case.get("classes", 1)
    if kind == "forest":
        sub = max(1, math.ceil(math.sqrt(f)))
        return {"bytes": trees * n * (sub + 1 + 8), "flops": 3 * trees * n * sub}
    width = 2 if case["bins"] > 256 else 1
    per_tree = cells * width + n * (8 + 16 + (8 if case.get("weighted") else 0))
    matrix = 4 * cells if kind in ("fit", "softmax") else 0
    return {"bytes": matrix + trees * per_tree + n * 8 * case.get("classes", 1), "flops": 3 * trees * cells}


# --------------------------------------------------------------------------------------
# The same calls in 64 bits
# --------------------------------------------------------------------------------------
def _quantile_bins(x: np.ndarray, max_bins: int):
    """Feature-major bins (missing rows at the feature's bin count) and bin counts of a
    row-major float32 matrix: boundaries at the quantile ranks, below the maximum and
    strictly increasing."""

    bins, counts = [], []
    for j in range(x.shape[1]):
        col = x[:, j]
        v = np.sort(col[~np.isnan(col)])
        m = v.size
        k = min(m, max_bins)
        bnd = np.empty(0, np.float32)
        if k > 1:
            part = np.arange(1, k, dtype=np.int64)
            rank = -(-part * m // k) - 1
            c = v[rank]
            bnd = np.unique(c[c < v[-1]])
        bins.append(np.where(np.isnan(col), bnd.size + 1, np.searchsorted(bnd, col, side="left")))
        counts.append(bnd.size + 1)
    return np.stack(bins), np.asarray(counts)


def _dataset_bins(ds):
    counts = ds.bin_counts.astype(np.int64)
    return np.where(ds.missing, counts[:, None], ds.bins.astype(np.int64)), counts


def _grow(bins: torch.Tensor, counts: torch.Tensor, g: torch.Tensor, h: torch.Tensor, depth: int,
          msl: int = 20, mcw: float = 1.0, lam: float = 1.0) -> torch.Tensor:
    """Level-wise tree of FP64 histograms; the leaf value of every row. Missing rows are
    tried left, then right; ties go to the lower feature and threshold, left first."""

    f, n = bins.shape
    width = int(counts.max()) + 1
    dev = bins.device
    node = torch.zeros(n, dtype=torch.int64, device=dev)
    value = (-g.sum() / (h.sum() + lam)).repeat(n)
    live = torch.ones(n, dtype=torch.bool, device=dev)
    ones = torch.ones_like(g)
    for level in range(depth):
        rows = torch.nonzero(live).squeeze(1)
        if rows.numel() == 0:
            break
        ids, node_of = torch.unique(node[rows], return_inverse=True)
        k = ids.numel()
        gain = torch.full((k,), -1.0, dtype=torch.float64, device=dev)
        pick = torch.zeros((k, 3), dtype=torch.int64, device=dev)
        stats = torch.stack([ones[rows], g[rows], h[rows]], 1)
        total = torch.zeros(k, 3, dtype=torch.float64, device=dev).index_add_(0, node_of, stats)

        def score(s):
            return s[..., 1] ** 2 / (s[..., 2] + lam)

        for j in range(f):
            c = int(counts[j])
            if c < 2:
                continue
            hist = torch.zeros(k * width, 3, dtype=torch.float64, device=dev)
            hist.index_add_(0, node_of * width + bins[j, rows], stats)
            hist = hist.view(k, width, 3)
            miss = hist[:, c]
            left = hist[:, : c - 1].cumsum(1)
            both = []
            for lost in (miss[:, None], torch.zeros_like(miss)[:, None]):
                l_side = left + lost
                r_side = total[:, None] - l_side
                s = 0.5 * (score(l_side) + score(r_side) - score(total)[:, None])
                ok = ((l_side[..., 0] >= msl) & (r_side[..., 0] >= msl) & (l_side[..., 2] >= mcw)
                      & (r_side[..., 2] >= mcw) & (s > 0))
                both.append(torch.where(ok, s, torch.full_like(s, -1.0)))
            s = torch.stack(both, 2).view(k, -1)  # (threshold, direction)
            best, at = s.max(1)
            better = best > gain
            gain = torch.where(better, best, gain)
            new = torch.stack([torch.full_like(at, j), at // 2, 1 - at % 2], 1)
            pick = torch.where(better[:, None], new, pick)
        split = gain > 0
        mine = split[node_of]
        keep = rows[mine]
        p = pick[node_of[mine]]
        b = bins[p[:, 0], keep]
        lost = b == counts[p[:, 0]]
        goes_left = torch.where(lost, p[:, 2] == 1, b <= p[:, 1])
        live = torch.zeros_like(live)
        live[keep] = True
        node[keep] = 2 * node[keep] + torch.where(goes_left, 1, 2)
        ids, node_of = torch.unique(node[keep], return_inverse=True)
        s = torch.zeros(ids.numel(), 2, dtype=torch.float64, device=dev)
        s.index_add_(0, node_of, torch.stack([g[keep], h[keep]], 1))
        value[keep] = (-s[:, 0] / (s[:, 1] + lam))[node_of]
    return value


def _boost_exact(case: dict, bins: np.ndarray, counts: np.ndarray, y: np.ndarray, w: np.ndarray | None) -> dict:
    dev = _device()
    b = torch.from_numpy(np.ascontiguousarray(bins, np.int64)).to(dev)
    c = torch.from_numpy(counts.astype(np.int64)).to(dev)
    yt = torch.from_numpy(y).to(dev)
    wt = torch.ones_like(yt) if w is None else torch.from_numpy(w).to(dev)
    if case["kind"] == "softmax":
        k = case["classes"]
        hot = torch.nn.functional.one_hot(yt.long(), k).double()
        base = torch.log(hot.mean(0).clamp_min(1e-15))
        m = base[None, :].repeat(y.size, 1)
        for _ in range(case["trees"]):
            for t in range(k):  # a class's margins move before the next class's tree
                p = torch.softmax(m, 1)[:, t]
                m[:, t] += 0.1 * _grow(b, c, p - hot[:, t], p * (1 - p), case["depth"])
        return {"base": base.cpu().numpy(), "predictions": m.cpu().numpy()}
    mean = float((yt * wt).sum() / wt.sum())
    base = math.log(mean / (1 - mean)) if case["objective"] == "binary_logistic" else mean
    m = torch.full_like(yt, base)
    for _ in range(case["trees"]):
        if case["objective"] == "binary_logistic":
            p = torch.sigmoid(m)
            g, h = p - yt, p * (1 - p)
        else:
            g, h = m - yt, torch.ones_like(m)
        m = m + 0.1 * _grow(b, c, g * wt, h * wt, case["depth"])
    return {"base": base, "predictions": m.cpu().numpy()}


def _score_exact(case: dict, seed: int) -> dict:
    train, x = _score_inputs(case, seed)
    rng = np.random.default_rng(seed)
    bounds = []
    for j in range(train.shape[1]):
        v = np.sort(train[:, j][~np.isnan(train[:, j])])
        k = min(v.size, case["bins"])
        c = v[-(-np.arange(1, k, dtype=np.int64) * v.size // k) - 1]
        bounds.append(np.unique(c[c < v[-1]]))
    counts = np.asarray([b.size + 1 for b in bounds], np.int64)
    trees = _random_trees(case, counts, rng)
    bins = np.stack([np.searchsorted(b, x[:, j], side="left") for j, b in enumerate(bounds)])
    dev = _device()
    bt = torch.from_numpy(bins).to(dev)
    lost = torch.from_numpy(np.isnan(x).T.copy()).to(dev)
    rows = torch.arange(x.shape[0], device=dev)
    out = torch.full((x.shape[0],), 0.25, dtype=torch.float64, device=dev)
    for t in trees:
        col = {k: torch.from_numpy(t[k].astype(np.int64)).to(dev)
               for k in ("feature_index", "threshold_bin", "left_child", "right_child", "default_left")}
        at = torch.zeros_like(rows)
        for _ in range(case["depth"]):
            f = col["feature_index"][at]
            left = torch.where(lost[f, rows], col["default_left"][at] != 0, bt[f, rows] <= col["threshold_bin"][at])
            at = torch.where(left, col["left_child"][at], col["right_child"][at])
        out += 0.1 * torch.from_numpy(t["leaf_value"].copy()).to(dev)[at]
    return {"predictions": out.cpu().numpy()}


def _layer_exact(case: dict, seed: int) -> dict:
    ds, pairs, rows = _layer_inputs(case, seed)
    dev = _device()
    bins = torch.from_numpy(ds.bins.astype(np.int64)).to(dev)  # a missing row is in bin 0
    p = torch.from_numpy(pairs).to(dev)
    out = []
    for r in rows:
        rt = torch.from_numpy(r.astype(np.int64)).to(dev)
        for j in range(ds.features):
            h = torch.zeros(int(ds.bin_counts[j]), 3, dtype=torch.float64, device=dev)
            h.index_add_(0, bins[j, rt], torch.cat([torch.ones_like(p[rt, :1]), p[rt]], 1))
            out.append(h)
    h = torch.cat(out).cpu().numpy()
    return {"count": h[:, 0].astype(np.int64), "gradient": h[:, 1], "hessian": h[:, 2]}


def exact(case: dict, seed: int):
    """What ``run`` returns, in 64 bits: predictions of the same boosting (a tree's nodes
    have no value of their own there), scores, histograms. None for fits whose plain
    restatement takes too long, leaf-wise growth and forests."""

    kind = case["kind"]
    if kind == "layer":
        return _layer_exact(case, seed)
    if kind == "score":
        return _score_exact(case, seed)
    if kind in ("ovr", "forest") or case.get("leaves"):
        return None
    trees = case["trees"] * case.get("classes", 1)
    if trees * case["depth"] * (case["features"] * (1.2e-3 + 2e-9 * case["rows"])) > 12.0:  # seconds, about
        return None
    if kind in ("fit", "softmax"):
        x, y, w = _fit_inputs(case, seed)
        bins, counts = _quantile_bins(x, case["bins"])
    else:
        ds, y, w = _boost_inputs(case, seed)
        bins, counts = _dataset_bins(ds)
    out = _boost_exact(case, bins, counts, y, w)
    return {"base": out["base"], "predictions": out["predictions"], "trees": None}
