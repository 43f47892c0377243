"""The native pass over class labels against the sort and search it replaces, and the result buffers beside
it (no GPU)."""

import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

from mpsboost_gb300 import build
from mpsboost_gb300.backend import _ResultBuffers
from mpsboost_gb300.estimators import _encode_classes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


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


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_class_ids_without_memory(tmp_path):
    lib = build.build()
    exe = tmp_path / "no_memory_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "native", "no_memory_check.cpp"), lib, "-rdynamic",
                    f"-Wl,-rpath,{os.path.dirname(lib)}", "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr


# Where no thread can be started, the training results' pages are mapped by the copy instead.
def test_result_buffers_without_a_thread(monkeypatch):
    def refuse(self):
        raise RuntimeError("can't start new thread")

    monkeypatch.setattr(threading.Thread, "start", refuse)
    results = _ResultBuffers(2, 600_000)
    results.join()
    for k in range(2):
        assert results[k].shape == (600_000,) and results[k].dtype == np.float64
    assert results[0] is not results[1]
