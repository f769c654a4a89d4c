"""The order of the service's copies between its streams (the autotuner's trials,
bursts of admissions), on the host: its objects linked with a runtime that runs
no kernels but keeps the streams' order (fake_cudart.hpp)."""
import subprocess

import pytest

from fake_runtime import build_with_fake_runtime


def test_no_copies_race(tmp_path):
    exe = build_with_fake_runtime(tmp_path, "serve_order_harness.cpp")
    if not exe:
        pytest.skip("no C++ compiler or no built objects")
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[:2000] + r.stderr
