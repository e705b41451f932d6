"""Side streams are joined however a launch sequence ends (host code, no GPU)."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dmhm_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_every_exit_joins(tmp_path):
    exe = tmp_path / "fork_scope_check"
    subprocess.run(["g++", "-std=c++17", "-I", CSRC,
                    os.path.join(ROOT, "tests", "cpp", "fork_scope_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_forks_go_through_the_scope():
    """fork() and join() are called by the scope alone, not around launches that may throw."""
    bad = [n for n in sorted(os.listdir(CSRC)) if n != "fork_scope.h" and re.search(
        r"ctx_?\.(fork|join)\(", open(os.path.join(CSRC, n)).read())]
    assert not bad, bad
