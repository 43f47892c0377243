"""The per-level kernels at the edges of their tiles, bit-exact to the oracle's fixed-point
replica (every tree node and training prediction)."""

from __future__ import annotations

import os
import subprocess
import threading

import numpy as np
import pytest

import mpsboost_gb300 as mb
import oracle
from conftest import seeded_matrix
from test_gpu_forest import _oracle_tree

pytestmark = pytest.mark.gpu


def assert_equals_replica(backend, port, x, y, w, max_bins, **params):
    model = mb.train_regressor(backend, mb.quantize_dense(x, max_bins), y, w, **params)
    ds = port.quantize_dense(x, max_bins)
    want = port.train_regressor(ds, y, w, hist_mode=oracle.HIST_FIXED, **params)
    assert [t.tobytes() for t in model.trees] == [t.tobytes() for t in want.trees]
    assert model.train_predictions.tobytes() == want.predict(ds).tobytes()


def targets(x, seed):
    rng = np.random.default_rng(seed)
    xs = np.nan_to_num(x)
    y = xs[:, 0] + xs[:, -1] * xs[:, x.shape[1] // 2] + rng.normal(size=x.shape[0]) * 0.2
    return y, rng.uniform(0.5, 1.5, x.shape[0])


# Bins around a warp's 64 slots, the page's 256 and the wide pages; feature counts around an
# item's 8 features and a block's 32; with and without the missing slot; a level-wise and a
# leaf-wise fit each (the sibling's histogram formed by the scan in both).
@pytest.mark.parametrize("bins,features,nan", [
    (2, 1, 0.0), (3, 7, 0.2), (63, 9, 0.0), (64, 8, 0.1), (65, 33, 0.1), (128, 31, 0.0),
    (255, 65, 0.05), (256, 12, 0.0), (256, 12, 0.1), (511, 5, 0.1), (512, 5, 0.1), (513, 9, 0.0),
])
@pytest.mark.parametrize("leaves", [0, 6])
def test_split_scan_edges(backend, port, bins, features, nan, leaves):
    x = seeded_matrix(bins + features, 3000, features, nan, integer_columns=features // 3)
    y, w = targets(x, bins)
    growth = dict(growth_strategy="leaf_wise", max_leaves=leaves) if leaves else {}
    assert_equals_replica(backend, port, x, y, w, bins, n_estimators=2, learning_rate=0.3, max_depth=5,
                          min_samples_leaf=4, min_child_weight=2.0, **growth)


# Nodes with up to 8 features to evaluate exactly, one more and all of them (equal columns tie;
# monotone constraints and hessians at min_child_weight take every feature), which a node's CTAs
# share from 33 features on; u8 and u16 pages, level-wise and leaf-wise.
@pytest.mark.parametrize("features,equal", [(32, 32), (33, 8), (33, 9), (70, 70), (260, 9), (1000, 300)])
@pytest.mark.parametrize("bins", [32, 300])
@pytest.mark.parametrize("leaves", [0, 6])
@pytest.mark.parametrize("extra", ["", "monotone", "hessian"])
def test_exact_scan_shared_by_ctas(backend, port, features, equal, bins, leaves, extra):
    x = seeded_matrix(features + equal, 1500, features, 0.05, integer_columns=3)
    rng = np.random.default_rng(equal)
    x[:, rng.choice(features, equal, replace=False)] = x[:, [features // 2]]
    y = np.nan_to_num(x[:, features // 2]) + rng.normal(size=1500) * 0.2
    params = dict(n_estimators=2, learning_rate=0.3, max_depth=4, min_samples_leaf=2)
    if extra == "monotone":
        params["monotonic_constraints"] = [1, 0, -1, 1] * (features // 4) + [0] * (features % 4)
    if extra == "hessian":
        params["min_child_weight"] = 20.0
    if leaves:
        params.update(growth_strategy="leaf_wise", max_leaves=leaves)
    assert_equals_replica(backend, port, x, y, None, bins, **params)


# Float histograms: the left sums are FP64 sums of the slots below. A slot of hessian 2e-5 beside
# one of 2e13 keeps its candidate (left hessian 2e-5 to the FP32 rounding of a row's pair), at
# even and odd slots, at a warp's and a page's edges and on u16 pages.
@pytest.mark.parametrize("bins,light", [(3, 0), (64, 1), (64, 62), (255, 63), (255, 64), (256, 254), (600, 255),
                                        (600, 256), (600, 598)])
@pytest.mark.parametrize("growth", [{}, dict(growth_strategy="leaf_wise", max_leaves=2)])
def test_float_left_sums_keep_small_slots(backend, bins, light, growth):
    b = np.repeat(np.arange(bins), 20)
    w = np.full(b.size, 1e-6)
    w[b == light + 1] = 1e12
    y = np.where(b == light, 1e6, 0.0)
    ds = mb.BinnedDataset(b.size, 1, bins, b[None].astype(np.uint16 if bins > 256 else np.uint8),
                          np.zeros((1, b.size), bool), np.arange(1, bins, dtype=np.float32), np.zeros(1, np.uint64),
                          np.array([bins - 1], np.uint32), np.array([bins], np.uint32), np.zeros(1, np.uint64))
    m = mb.train_regressor(backend, ds, y, w, hist_mode="float", n_estimators=1, max_depth=1, reg_lambda=1e-3, **growth)
    g = w * (m.base_score - y)
    left = b <= light
    root = m.trees[0][0]
    assert (root["flags"] & 1) == 0 and root["threshold_bin"] == light
    # 20 rows of FP32 pairs added in FP32: 21 roundings of 2^-24, twice.
    np.testing.assert_allclose(m.trees[0][root["left_child"]]["leaf_value"],
                               -g[left].sum() / (w[left].sum() + 1e-3), rtol=1e-5)


# Leaf-wise trees of several classes: the step that chooses and splits a leaf takes a warp per
# tree, eight at a time, so class counts below, at and past that; each class's trees are those
# of a fit of the class alone. A depth limit frees slots, an interaction list writes the paths.
@pytest.mark.parametrize("classes", [2, 8, 9, 17])
@pytest.mark.parametrize("extra", [{}, dict(max_depth=3), dict(interaction_constraints=[[0, 1, 2], [2, 3, 4, 5]])])
def test_leafwise_classes_equal_single_fits(backend, classes, extra):
    x = seeded_matrix(classes, 5000, 6, 0.05, integer_columns=2)
    rng = np.random.default_rng(classes)
    y = (np.argsort(np.argsort(np.nan_to_num(x[:, 0]) + rng.normal(size=5000) * 0.5)) * classes // 5000).astype(float)
    binned = mb.quantize_dense(x, 64)
    params = dict(n_estimators=2, learning_rate=0.3, max_depth=7, min_samples_leaf=2, objective="binary_logistic",
                  growth_strategy="leaf_wise", max_leaves=20)
    params.update(extra)
    got = mb.train_ovr(backend, binned, y, classes, **params)
    for k, m in enumerate(got):
        want = mb.train_regressor(backend, binned, (y == k).astype(float), **params)
        assert [t.tobytes() for t in m.trees] == [t.tobytes() for t in want.trees]
        assert m.train_predictions.tobytes() == want.train_predictions.tobytes()


# Rows around the 32-row flag words, a CTA's 1,024 rows, 16 CTAs of a cluster and their
# 48 rows per thread (786,432: the last single-launch partition of a root, and one past it).
@pytest.mark.parametrize("rows", [33, 511, 1025, 16 * 1024 - 1, 16 * 1024 + 1, 70_001, 786_432, 786_433])
def test_partition_edges(backend, port, rows):
    x = seeded_matrix(rows, rows, 3, 0.05, integer_columns=1)
    y, w = targets(x, rows)
    assert_equals_replica(backend, port, x, y, w, 64, n_estimators=2, learning_rate=0.3, max_depth=4,
                          min_samples_leaf=2)


# The cluster partition at the largest nodes that it takes: 16 rows a thread of 16 CTAs for a root
# (262,144 rows; one more takes the three launches), twice that from four nodes on, where a node
# may hold nearly all rows, and in leaf-wise steps up to the flag words of 16 CTAs.
@pytest.mark.parametrize("rows,growth", [
    (262_144, {}), (262_145, {}), (524_288, {}), (524_289, {}),
    (1_048_576, dict(growth_strategy="leaf_wise", max_leaves=4)),
    (1_048_577, dict(growth_strategy="leaf_wise", max_leaves=4)),
])
def test_partition_largest_nodes(backend, port, rows, growth):
    x = seeded_matrix(rows, rows, 2, 0.05)
    x[:, 1] = np.arange(rows) % 997 < 2  # nearly all rows in one child, level by level
    rng = np.random.default_rng(rows)
    y = 5.0 * x[:, 1] + 0.1 * np.nan_to_num(x[:, 0]) + (x[:, 0] > 2.5) * 3.0 + rng.normal(size=rows) * 0.05
    assert_equals_replica(backend, port, x, y, None, 32, n_estimators=1, learning_rate=0.3, max_depth=4,
                          min_samples_leaf=2, **growth)


# A histogram cell of 2,047 rows (the packed limbs' largest), one past it, and multiples of
# 2,048 (whose count fields read 0), in a block with continuous features; unweighted fits
# build two packed words, weighted ones four.
@pytest.mark.parametrize("heavy", [2047, 2048, 4096, 6144])
@pytest.mark.parametrize("weighted", [False, True])
def test_packed_limb_overflow(backend, port, heavy, weighted):
    x = seeded_matrix(heavy, 10_000, 34, 0.0)
    x[:, 1] = 1.0
    x[:heavy, 1] = 0.0
    x[:, 33] = np.arange(10_000) % 3 == 0
    y, w = targets(x, heavy)
    assert_equals_replica(backend, port, x, y, w if weighted else None, 255, n_estimators=3, learning_rate=0.3,
                          max_depth=4, min_samples_leaf=2)


# Wide pages: the packed limbs' largest cells (127 rows weighted, 2,047 unweighted) and one past
# them, missing rows in most and in few cells, few-valued features whose passes fall back to split
# limbs, and passes of 32, 16 and 8 features (weighted, 512 / 1,024 / 2,048 slots) at feature
# counts around a pass and a block; past 2,133 slots the split limbs alone.
@pytest.mark.parametrize("bins,features", [(300, 33), (511, 7), (700, 17), (1000, 40), (2000, 9), (2200, 5)])
@pytest.mark.parametrize("heavy,nan", [(127, 0.0), (128, 0.3), (2047, 0.0), (2048, 0.02)])
@pytest.mark.parametrize("weighted", [False, True])
def test_wide_packed_limbs(backend, port, bins, features, heavy, nan, weighted):
    x = seeded_matrix(bins + heavy, 9_000, features, nan)
    x[:, 1] = np.arange(9_000)
    x[:heavy, 1] = -1.0
    x[:, features - 1] = np.arange(9_000) % 3
    y, w = targets(x, heavy)
    assert_equals_replica(backend, port, x, y, w if weighted else None, bins, n_estimators=2, learning_rate=0.3,
                          max_depth=4, min_samples_leaf=2)


def test_integer_pipe_logistic_within_half_an_ulp(tmp_path):
    """e^-t and the logistic function's pieces on the integer pipe against long double."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    exe = tmp_path / "logistic_check"
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-I", os.path.join(root, "mpsboost_gb300", "csrc"), "-I", os.path.join(root, "include"),
                    os.path.join(root, "tests", "native", "logistic_check.cu"), "-o", str(exe)],
                   check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout + run.stderr


# Unweighted class fits count their labels on the device: rows around a CTA's 1,024 and a
# label that is no class id.
@pytest.mark.parametrize("rows", [40, 1023, 1025, 300_001])
@pytest.mark.parametrize("classes", [2, 7])
def test_class_counts_give_the_base_scores(backend, rows, classes):
    x = seeded_matrix(rows, rows, 2)
    y = np.random.default_rng(rows).integers(0, classes, rows).astype(np.float64)
    y[:classes] = np.arange(classes)
    binned = mb.quantize_dense(x, 16)
    params = dict(n_estimators=1, max_depth=2, learning_rate=0.5)
    share = [np.count_nonzero(y == k) / rows for k in range(classes)]
    got = [m.base_score for m in mb.train_ovr(backend, binned, y, classes, **params)]
    np.testing.assert_allclose(got, [np.log(p / (1 - p)) for p in share], rtol=1e-15, atol=1e-15)
    soft = mb.train_softmax(backend, binned, y, classes, **params)
    np.testing.assert_allclose(soft.base_scores, np.log(share), rtol=1e-15)
    y[-1] = 0.5
    with pytest.raises(mb.TrainingError, match="0 or 1" if classes == 2 else "class ids"):
        if classes == 2:
            mb.train_regressor(backend, binned, y, objective="binary_logistic", **params)
        else:
            mb.train_softmax(backend, binned, y, classes, **params)


# Forest trees on copies of their own features: subsets around a 32-feature block and the
# half of the dataset's 70 from which the copy is made, ragged between trees; rows around
# an expansion chunk's 4,096 and the pack's words; rows drawn 0, many and 255 times; random
# thresholds and monotone constraints count the tree's and the dataset's features.
@pytest.mark.parametrize("rows", [4095, 4097, 8192])
@pytest.mark.parametrize("subset,extra", [(1, {}), (31, {}), (33, dict(split_strategy="random_threshold")),
                                          (35, dict(monotonic_constraints=[1, 0, -1, 0, 0] * 14)), (36, {})])
@pytest.mark.parametrize("weighted", [False, True])
def test_compact_forest_equals_replica(backend, port, rows, subset, extra, weighted):
    x = seeded_matrix(rows + subset, rows, 70, 0.05, integer_columns=9)
    y, w = targets(x, subset)
    w = w if weighted else None
    rng = np.random.default_rng(subset)
    counts = rng.poisson(0.8, (3, rows)).astype(np.uint8)
    counts[0, 5], counts[1, :2000] = 255, 0
    subsets = [rng.choice(70, max(1, subset - 2 * t), replace=False) for t in range(3)]
    seeds = np.arange(3, dtype=np.uint32)
    params = dict(max_depth=5, min_samples_leaf=3, **extra)
    binned = mb.quantize_dense(x, 64)
    models = mb.train_forest(backend, binned, y, w, row_counts=counts, feature_subsets=subsets, seeds=seeds, **params)
    ds = port.quantize_dense(x, 64)
    for t, m in enumerate(models):
        p = dict(params)
        if "monotonic_constraints" in p:
            p["monotonic_constraints"] = [p["monotonic_constraints"][f] for f in np.sort(subsets[t])]
        base, nodes = _oracle_tree(port, ds, y, w, counts[t], subsets[t], p, seeds[t])
        assert float(m.base_score).hex() == float(base).hex()
        assert m.trees[0].tobytes() == nodes.tobytes()


# Subsets shorter than the widest pad a tree's block with a feature that holds all rows in one
# bin, past the packed limbs' cells; heavy cells in features that the tree has and has not, in
# copies of its own features (8 of 70) and in the dataset's (68 of 70).
@pytest.mark.parametrize("widest", [8, 68])
@pytest.mark.parametrize("weighted", [False, True])
def test_forest_packed_limbs_of_ragged_subsets(backend, port, widest, weighted):
    x = seeded_matrix(widest, 9_000, 70, 0.0)
    x[:, 0] = np.arange(9_000) < 2_048
    x[:, 5] = np.arange(9_000) % 2
    y, w = targets(x, widest)
    w = w if weighted else None
    rng = np.random.default_rng(widest)
    counts = rng.poisson(1.0, (4, 9_000)).astype(np.uint8)
    subsets = [rng.choice(np.arange(6, 70) if t % 2 else 70, s, replace=False)
               for t, s in enumerate([widest, min(widest - 1, 64), widest - 4, 1])]
    params = dict(max_depth=6, min_samples_leaf=3)
    models = mb.train_forest(backend, mb.quantize_dense(x, 255), y, w, row_counts=counts, feature_subsets=subsets, **params)
    ds = port.quantize_dense(x, 255)
    for t, m in enumerate(models):
        base, nodes = _oracle_tree(port, ds, y, w, counts[t], subsets[t], params, 0)
        assert float(m.base_score).hex() == float(base).hex()
        assert m.trees[0].tobytes() == nodes.tobytes()


def _traverse(trees, lr, base, bins, missing):
    """Predictions tree by tree in FP64, as RegressionModel::Predict adds them."""
    out = np.full(bins.shape[1], base)
    rows = np.arange(bins.shape[1])
    for t in trees:
        at = np.zeros(rows.size, np.int64)
        for _ in range(t.size):
            f = t["feature_index"][at]
            left = np.where(missing[f, rows], t["default_left"][at] != 0, bins[f, rows] <= t["threshold_bin"][at])
            step = np.where(left, t["left_child"][at], t["right_child"][at]).astype(np.int64)
            leaf = (t["flags"][at] & 1) != 0
            if leaf.all():
                break
            at = np.where(leaf, at, step)
        out = out + lr * t["leaf_value"][at]
    return out


def _grown(rng, features, bins, splits, shuffle):
    """A tree grown by splitting a random leaf at a time; shuffled, children may precede
    their parents."""
    n = 2 * splits + 1
    t = np.zeros(n, mb._lib.NODE_DTYPE)
    t["flags"] = 1
    t["leaf_value"] = rng.normal(size=n)
    leaves, used = [0], 1
    for _ in range(splits):
        at = leaves.pop(rng.integers(len(leaves)))
        t["flags"][at] = 0
        t["feature_index"][at], t["threshold_bin"][at] = rng.integers(features), rng.integers(bins)
        t["default_left"][at] = rng.integers(2)
        t["left_child"][at], t["right_child"][at] = used, used + 1
        leaves += [used, used + 1]
        used += 2
    if shuffle:
        order = np.concatenate([[0], 1 + rng.permutation(n - 1)])  # new index of each node
        u = np.empty_like(t)
        u[order] = t
        inner = (u["flags"] & 1) == 0
        u["left_child"][inner], u["right_child"][inner] = order[u["left_child"][inner]], order[u["right_child"][inner]]
        t = u
    return t


# Rows around a CTA's 128 and the staged words, features up to and past the staging, trees
# of one leaf, of groups' size (4,096 nodes) and past it, u8 and u16 bins, missing rows; and
# a tree whose children precede their parents, which the general kernel walks.
@pytest.mark.parametrize("rows,features,bins,nan,splits,shuffle", [
    (1, 1, 4, 0.0, [0, 1], False), (127, 5, 64, 0.2, [3, 0, 40], False), (129, 33, 255, 0.1, [63] * 70, False),
    (1000, 64, 255, 0.1, [200] * 9, False), (2050, 12, 256, 0.1, [50] * 5, False),
    (3001, 7, 900, 0.1, [500, 30], False), (400, 6, 128, 0.1, [4095, 10, 4096 - 10], False),
    (400, 6, 128, 0.1, [4097], False), (300, 1300, 32, 0.0, [60], False), (500, 8, 64, 0.1, [30, 31], True),
])
def test_predict_edges(backend, rows, features, bins, nan, splits, shuffle):
    rng = np.random.default_rng(rows)
    binned = mb.quantize_dense(seeded_matrix(rows, max(rows, 2), features, nan), bins)
    trees = [_grown(rng, features, max(2, bins - 2), s, shuffle) for s in splits]
    model = mb.RegressionModel(0.25, 0.1, trees)
    got = model.predict(backend, binned)
    assert got.tobytes() == _traverse(trees, 0.1, 0.25, binned.bins, binned.missing).tobytes()


# Both prediction kernels around the rule that chooses between them: 32 KB of bins a CTA and one
# feature more with few visits, four bytes a visit and more, features that halve and quarter a
# CTA's rows with few and many trees, trees in groups of the staging's 4,096 nodes on few rows
# and on many, u8 and u16 bins.
@pytest.mark.parametrize("rows,features,bins,splits", [
    (5_000, 256, 32, [63]), (5_000, 257, 32, [63]), (20_000, 264, 32, [63] * 11), (20_000, 265, 32, [63] * 11),
    (160_001, 200, 32, [15] * 3), (160_001, 200, 32, [15] * 90), (160_000, 400, 32, [15] * 90),
    (2_000, 6, 64, [4000, 90, 10, 4096]), (160_002, 6, 64, [4000, 90, 10, 4096]), (160_003, 70, 300, [31] * 40),
    (160_003, 130, 300, [31] * 40),
])
def test_predict_routes(backend, rows, features, bins, splits):
    rng = np.random.default_rng(features)
    counts = np.full(features, bins, np.uint32)
    b = rng.integers(0, bins, (features, rows)).astype(np.uint16 if bins > 256 else np.uint8)
    binned = mb.BinnedDataset(rows, features, bins, b, np.zeros(b.shape, bool),
                              np.tile(np.arange(1, bins, dtype=np.float32), features),
                              np.arange(features, dtype=np.uint64) * (bins - 1), counts - 1, counts,
                              np.zeros(features, np.uint64))
    trees = [_grown(rng, features, bins - 1, s, False) for s in splits]
    got = mb.RegressionModel(0.25, 0.1, trees).predict(backend, binned)
    assert got.tobytes() == _traverse(trees, 0.1, 0.25, binned.bins, binned.missing).tobytes()


# Working memory kept between calls: fits of sizes that share, outgrow and split the kept blocks
# give the same bytes again, on one backend and on two threads with one each; 600,000 rows also
# take the result buffers mapped beside the training.
@pytest.mark.parametrize("threads", [1, 2])
def test_kept_memory_changes_nothing(threads):
    shapes = [(600_000, 5, 255), (3_000, 70, 255), (40_000, 9, 700), (1_000, 3, 16), (45_000, 9, 700)]
    data = []
    for rows, features, bins in shapes:
        x = seeded_matrix(rows, rows, features, 0.05)
        data.append((x, *targets(x, rows), bins))

    def fits(out):
        b = mb.CudaBackend(0)
        for _ in range(2):
            for x, y, w, bins in data:
                binned = mb.quantize_device(b, x, bins)
                m = mb.train_regressor(b, binned, y, w, n_estimators=2, max_depth=4)
                forest = mb.train_forest(b, binned, y, row_counts=np.ones((3, y.size), np.uint8),
                                         feature_subsets=[np.array([0]), np.array([1, 2]), np.array([0, 2])], max_depth=3)
                np.testing.assert_array_equal(m.train_predictions, m.predict(b, binned))
                out.append((m.train_predictions.tobytes(), [t.tobytes() for f in [m, *forest] for t in f.trees]))
                binned.close()

    outs = [[] for _ in range(threads)]
    pool = [threading.Thread(target=fits, args=(o,)) for o in outs]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    for o in outs:
        assert len(o) == 2 * len(data) and o == outs[0] and o[: len(data)] == o[len(data):]


def test_kept_memory_is_given_back(backend):
    torch = pytest.importorskip("torch")
    x = seeded_matrix(3, 200_000, 12)
    y, w = targets(x, 3)
    binned = mb.quantize_dense(x, 255)
    params = dict(n_estimators=2, max_depth=5)
    want = mb.train_regressor(backend, binned, y, w, **params)
    free = torch.cuda.mem_get_info(0)[0]
    given = backend.release_memory()
    assert 0 < given <= 8 << 30
    assert torch.cuda.mem_get_info(0)[0] - free >= given // 2
    assert backend.release_memory() == 0
    got = mb.train_regressor(backend, binned, y, w, **params)
    assert [t.tobytes() for t in got.trees] == [t.tobytes() for t in want.trees]


# Sessions that another thread drops (as a garbage collector may) while this one captures and runs
# rounds on the same backend: their memory goes back without waiting on a stream being captured.
def test_sessions_dropped_beside_a_capture(backend):
    x = seeded_matrix(9, 4_000, 8, 0.0)
    y, _ = targets(x, 9)
    binned = mb.quantize_dense(x, 64)
    params = dict(n_estimators=3, max_depth=4)
    want = [t.tobytes() for t in mb.train_regressor(backend, binned, y, **params).trees]
    idle = [mb.Trainer(backend, binned, y, **params) for _ in range(200)]
    dropper = threading.Thread(target=lambda: [t.close() for t in idle])
    dropper.start()
    rounds = 0
    while dropper.is_alive() or rounds < 20:
        got = mb.train_regressor(backend, binned, y, **params)
        assert [t.tobytes() for t in got.trees] == want
        rounds += 1
    dropper.join()


# Node-level calls convert their inputs and results on the device: row sets around a warp and a
# CTA, few-valued and missing features on u8 and u16 pages, bit-exact to the replica; the first
# error in the checks' order, rows before pairs, and scales of tiny and of zero pairs.
@pytest.mark.parametrize("bins", [5, 255, 700])
@pytest.mark.parametrize("rows", [1, 31, 257, 70_001])
@pytest.mark.parametrize("scale", [1.0, 1e-30, 0.0])
def test_node_histograms_edges(backend, port, bins, rows, scale):
    n = 70_001
    x = seeded_matrix(bins, n, 35, 0.1, 6)
    binned, ds = mb.quantize_dense(x, bins), port.quantize_dense(x, bins)
    rng = np.random.default_rng(rows)
    pairs = np.column_stack([rng.normal(size=n), rng.uniform(0.0, 2.0, n)]) * scale
    sel = rng.permutation(n)[:rows]
    p32 = pairs.astype(np.float32)
    kg, kh = port.fixed_scales(p32)
    want, miss = port.fixed_histograms(ds, p32, kg, kh, sel)
    for got in backend.layer_histograms(binned, pairs, [sel, sel]):
        for f, (gf, wf) in enumerate(zip(got, want)):
            total = {k: wf[k].copy() for k in ("count", "gradient_q", "hessian_q")}
            for k in total:
                total[k][0] += miss[f][k]
            np.testing.assert_array_equal(gf["count"], total["count"])
            np.testing.assert_array_equal(gf["gradient_sum"], total["gradient_q"].astype(np.float64) * 2.0 ** -kg)
            np.testing.assert_array_equal(gf["hessian_sum"], total["hessian_q"].astype(np.float64) * 2.0 ** -kh)


def test_node_histogram_errors_keep_their_order(backend):
    binned = mb.quantize_dense(seeded_matrix(1, 300, 3), 16)
    pairs = np.ones((300, 2))
    def bad(at, value):
        p = pairs.copy()
        p[at] = value
        return p
    for p, rows, match in [(bad((7, 1), -1.0), [1, 300], "out of bounds"), (bad((7, 1), -1.0), [1], "non-negative"),
                           (bad((299, 0), np.nan), [1], "finite"), (bad((0, 0), 1e39), [1], "float32 range"),
                           (bad((0, 0), 1e39), [1, 2**40], "out of bounds")]:
        with pytest.raises(mb.TrainingError, match=match):
            backend.layer_histograms(binned, p, [rows])
