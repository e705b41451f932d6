"""The reflectors' reciprocal against CUDA's correctly rounded one: at most one
unit in the last place (the rounding of its last multiply-add, less than one
unit from 1 / x, and half a unit of the other's)."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.mark.skipif(shutil.which(NVCC) is None, reason="no nvcc")
def test_reciprocal_is_within_one_unit(tmp_path):
    exe = tmp_path / "reciprocal_check"
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-I", os.path.join(ROOT, "dmhm_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "reciprocal_check.cu"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    assert 0.0 <= float(r.stdout) <= 1.0, r.stdout
