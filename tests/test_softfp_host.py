"""The core of the step kernel's integer-pipe binary64 arithmetic
(fv2d_gb300/csrc/softfp.cuh), compiled for the host: division, square root and
multiplication must give the host's bits for random significands, significands
with few set bits, next to a power of two and with runs at the digit
boundaries, over every exponent, and operands next to exact quotients, products
and perfect squares -- with the FP32 seeds exact and moved by up to three units
in the last place, more than the device's approximations are off."""
import os
import shutil
import subprocess

import pytest

from fv2d_testlib import REPO


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    cxx = shutil.which(os.environ.get("CXX", "g++")) or shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("softfp") / "softfp_harness")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-Wno-unused-function", "-ffp-contract=off",
                    "-o", exe, os.path.join(REPO, "tests", "softfp_harness.cpp")], check=True)
    return exe


@pytest.mark.parametrize("ulps", [-3, -1, 0, 1, 3])
def test_core_arithmetic_matches_the_host(harness, ulps):
    r = subprocess.run([harness, "2000000", str(1000 + ulps), str(ulps)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "0", r.stdout
