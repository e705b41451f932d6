"""Block structures are told apart by an id that is never given out again (host
code, no GPU): plans and work lists outlive the matrix they were made for, and
a structure's address does not."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dmhm_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_ids_are_unique(tmp_path):
    exe = tmp_path / "structure_id_check"
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", cuda_inc,
                    os.path.join(ROOT, "tests", "cpp", "structure_id_check.cpp"),
                    os.path.join(CSRC, "structure.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_no_cache_keeps_a_structure_by_address():
    bad = [n for n in sorted(os.listdir(CSRC)) if re.search(
        r"const Structure\s*\*\s*\w+\s*=\s*(nullptr|\w+(\.|->)S\.get\(\))",
        open(os.path.join(CSRC, n)).read())]
    assert not bad, bad
