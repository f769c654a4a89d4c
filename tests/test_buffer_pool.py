"""The memory that the service keeps for its results (BufferPool), on the host."""
import os
import shutil
import subprocess

import pytest

from fv2d_testlib import REPO


def test_the_oldest_buffers_go(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++")) or shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "buffers")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-pthread", "-o", exe,
                    os.path.join(REPO, "tests", "buffer_pool_harness.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
