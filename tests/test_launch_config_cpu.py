"""The launch shapes the autotuner tries (launch_config.h): no two of a field are the same launch; compiled
for the host."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_values_are_different_launches(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ is not available")
    exe = str(tmp_path / "launch_config_check")
    cmd = [cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "blend2d_gb300", "csrc"),
           os.path.join(HERE, "native", "launch_config_check.cpp"), "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout + res.stderr
