"""Sizing of the rounding kernels (host code, no GPU): the shared-memory layout
of the register form covers every op that is sent to it."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_layout_covers_every_op(tmp_path):
    exe = tmp_path / "round_sizing_check"
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "dmhm_b200", "csrc"), "-I", cuda_inc,
                    os.path.join(ROOT, "tests", "cpp", "round_sizing_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
