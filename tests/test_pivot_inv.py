"""pivot_inv, the branch-free reciprocal of the spline sweeps, equals 1.0/x bit for bit."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu


def test_pivot_inv_is_the_ieee_reciprocal(cuda, tmp_path):
    here = os.path.dirname(os.path.abspath(__file__))
    exe = str(tmp_path / "pivot_inv_check")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-O2", "-std=c++17", "-fmad=false", "-o", exe,
                    os.path.join(here, "pivot_inv_check.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split() == ["mismatches", "0"]
