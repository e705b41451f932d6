"""Kernel attributes belong to one device's copy of a kernel (host code, no
GPU): a context on a second device needs its own shared-memory limit and
occupancy, and a refused limit must be reported."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dmhm_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_records_are_kept_by_device(tmp_path):
    exe = tmp_path / "kernel_limits_check"
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", cuda_inc,
                    os.path.join(ROOT, "tests", "cpp", "kernel_limits_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_every_kernel_attribute_goes_through_the_record():
    """No source sets an attribute or caches an occupancy by itself (a
    process-wide once_flag would serve the first device only)."""
    bad = []
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        if name != "kernel_limits.h" and re.search(
                r"cudaFuncSetAttribute|cudaOccupancyMaxActive|std::once_flag", text):
            bad.append(name)
    assert not bad, bad
