"""Division of a correlator launch into work groups
(mflib_gb300/csrc/work_groups.h), on the host."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CXX = shutil.which("g++")


@pytest.mark.skipif(CXX is None, reason="g++ not found")
def test_work_groups(tmp_path):
    exe = str(tmp_path / "test_work_groups")
    r = subprocess.run([CXX, "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror",
                        "-I", os.path.join(ROOT, "mflib_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "test_work_groups.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    run = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr
