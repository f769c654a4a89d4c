"""The service's host threads and result buffers (fv2d_gb300/csrc/host_pool.hpp), on the host."""
import os
import shutil
import subprocess

import pytest

from fv2d_testlib import REPO


def test_parallel_loops_and_buffers(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++")) or shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "pool")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-pthread", "-o", exe,
                    os.path.join(REPO, "tests", "host_pool_harness.cpp")], check=True)
    assert subprocess.run([exe], timeout=120).returncode == 0
