"""The per-level kernels at the edges of their tiles, bit-exact to the oracle's fixed-point
replica (every tree node and training prediction)."""

from __future__ import annotations

import numpy as np
import pytest

import mpsboost_gb300 as mb
import oracle
from conftest import seeded_matrix

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


# Rows around the 32-row flag words, a CTA's 1,024 rows, 16 CTAs of a cluster and their
# 48 rows per thread (786,432: the last single-launch partition of a root, and one past it).
@pytest.mark.parametrize("rows", [33, 511, 1025, 16 * 1024 - 1, 16 * 1024 + 1, 70_001, 786_432, 786_433])
def test_partition_edges(backend, port, rows):
    x = seeded_matrix(rows, rows, 3, 0.05, integer_columns=1)
    y, w = targets(x, rows)
    assert_equals_replica(backend, port, x, y, w, 64, n_estimators=2, learning_rate=0.3, max_depth=4,
                          min_samples_leaf=2)
