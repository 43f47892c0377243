"""The native pass over class labels against the sort and search it replaces (no GPU)."""

import numpy as np
import pytest

from mpsboost_gb300.estimators import _encode_classes


# Class ids that are their own positions, gaps, the table's last number and one past it, a sign,
# a minus zero, a fraction; row counts around a thread's 2^17.
@pytest.mark.parametrize("rows", [5, 4097, (1 << 18) + 3])
@pytest.mark.parametrize("values", [[0, 1], [0, 1, 2, 9], [1, 2], [0, 4095], [0, 4096], [-1, 1], [-0.0, 1], [0, 0.5, 1],
                                    [0, 1e300]])
def test_class_positions(rows, values):
    y = np.random.default_rng(rows).choice(np.asarray(values, np.float64), rows)
    y[-len(values):] = values
    classes, encoded = _encode_classes(y)
    want = np.unique(y)
    np.testing.assert_array_equal(classes, want)
    np.testing.assert_array_equal(encoded, np.searchsorted(want, y).astype(np.float64))
    assert classes.dtype == want.dtype and encoded.dtype == np.float64
