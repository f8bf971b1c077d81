"""CPU: the table of memory pools by device and context
(csrc/host/context_table.h), in a host program."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_contexts_that_take_turns(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    exe = tmp_path / "context_table.bin"
    r = subprocess.run([cxx, "-O1", "-std=c++17", "-Wall", "-Werror",
                        f"-I{ROOT}/sparse-blas_b200/csrc/host",
                        os.path.join(ROOT, "tests", "c", "context_table_test.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
