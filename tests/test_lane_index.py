"""CPU: the index arithmetic of the lanes (csrc/kernels/lane_index.cuh) at the
limits of nnz, in a host program."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_lane_index_limits(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    exe = tmp_path / "lane_index.bin"
    r = subprocess.run([cxx, "-O1", "-std=c++17", "-Wall", "-Werror",
                        f"-I{ROOT}/sparse-blas_b200/csrc/kernels",
                        os.path.join(ROOT, "tests", "c", "lane_index_test.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
