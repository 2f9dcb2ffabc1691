"""The edge records of the bins: wherever crossing_f32 decides a crossing
from a record, as a pixel row evaluates it, it is the rounded f64 value, on
random and adversarial edges (tests/bin_edge_check.cu, built with nvcc
as host code and run on the CPU)."""
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_bin_records_match_f64():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "bin_edge_check")
        subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17",
                        "-Xcompiler", "-ffp-contract=off",
                        "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "z2d_gb300", "csrc"),
                        os.path.join(HERE, "bin_edge_check.cu"), "-o", exe], check=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "wrong 0" in r.stdout, r.stdout
