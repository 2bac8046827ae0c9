"""CPU test of the side branch of a context's stream (csrc/fk_branch.h):
branch_check.cpp makes each of its calls fail in turn."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_failed_fork_and_join(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "branch_check")
    subprocess.check_call([cxx, "-std=c++17", "-O1", "-Wall", "-Werror",
                           "-I", os.path.join(ROOT, "fortkernels-_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "branch_check.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
