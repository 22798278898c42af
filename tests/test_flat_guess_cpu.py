"""The tree flattener's 32-bit flatness test (eb::flat_guess) against the FP64 test it stands for, on
every node of random cubic and quadratic pieces inside the clip box, 1 to 65,535 px in size, on and off
the pixel grid: where it decides it decides alike, and it leaves few nodes open. Compiled for the host
from the device header."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ is not available")
    exe = str(tmp_path_factory.mktemp("flat") / "flat_guess_check")
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    cmd = [cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "blend2d_gb300", "csrc"), "-I",
           cuda_inc, os.path.join(HERE, "native", "flat_guess_check.cpp"), "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    return exe


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_decides_like_fp64(checker, seed):
    res = subprocess.run([checker, str(seed), "60000"], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
    assert "differ 0" in res.stdout
