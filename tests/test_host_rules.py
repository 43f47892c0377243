"""The rules that kernels and their host code share, on the host (no GPU)."""

from __future__ import annotations

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None and not os.path.exists("/usr/local/cuda/bin/nvcc"),
                    reason="no nvcc")
def test_host_rules(tmp_path):
    exe = tmp_path / "host_rules_check"
    subprocess.run([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-O1", "-std=c++17", "-I", os.path.join(ROOT, "mpsboost_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "native", "host_rules_check.cu"),
                    "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr
