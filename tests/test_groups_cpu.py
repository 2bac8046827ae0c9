"""CPU test of how a unit's stages are split into accumulator groups and chunks
(csrc/fk_groups.h): groups_check.cpp walks them as the MMA issuer and the epilogue do."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_groups_and_chunks(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "groups_check")
    subprocess.check_call([cxx, "-std=c++17", "-O1", "-Wall", "-Werror",
                           "-I", os.path.join(ROOT, "fortkernels-_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "groups_check.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
