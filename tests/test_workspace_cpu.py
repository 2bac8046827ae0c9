"""CPU test of the workspace's growth and of the choice between a request's two
workspace sizes (csrc/fk_workspace.h): workspace_check.cpp drives both with an
allocator that refuses."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_refused_growth_falls_back(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "workspace_check")
    subprocess.check_call([cxx, "-std=c++17", "-O1", "-Wall", "-Werror",
                           "-I", os.path.join(ROOT, "fortkernels-_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "workspace_check.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
