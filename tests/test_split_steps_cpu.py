"""Curves split into monotonic pieces in the steps a warp's lanes share (edge_build.cuh: curve_poly,
cubic_candidates, poly_piece) against split_cubic and split_quad, bit for bit; compiled for the host from
the device header."""
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
    exe = str(tmp_path_factory.mktemp("split") / "split_steps_check")
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    cmd = [cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "blend2d_gb300", "csrc"), "-I",
           cuda_inc, os.path.join(HERE, "native", "split_steps_check.cpp"), "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    return exe


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_steps_give_the_same_pieces(checker, seed):
    res = subprocess.run([checker, str(seed), "200000"], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
    assert "mismatches 0" in res.stdout
