"""The device's closed-form cell rasterizer (raster.cuh), compiled for the host, against the oracle's
banded DDA (pinned to the reference's cell grids): every window of random lines of all slopes and
directions, on whole-pixel and half-pixel coordinates and up to 65,535 px, with reciprocals off by
up to 3 ulp."""
import os
import shutil
import subprocess

import pytest

import oracle_lib

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ is not available")
    oracle_lib.lib()                         # built
    exe = str(tmp_path_factory.mktemp("rows") / "raster_rows_check")
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    build = os.path.join(ROOT, "oracle", "_build")
    cmd = [cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "blend2d_gb300", "csrc"), "-I",
           os.path.join(ROOT, "oracle"), "-I", cuda_inc, os.path.join(HERE, "native", "raster_rows_check.cpp"), "-o",
           exe, os.path.join(build, "liboracle.so"), f"-Wl,-rpath,{build}"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    return exe


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_rows_match_the_banded_rasterizer(checker, seed):
    res = subprocess.run([checker, str(seed), "30000"], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
    assert "mismatches 0" in res.stdout
