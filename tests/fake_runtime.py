"""Builds a host harness from the library's objects and fake_cudart.hpp."""
import glob
import os
import shutil
import subprocess

from fv2d_testlib import REPO

UNITS = ("fv2d_api", "serve", "batch_kernels", "batch_march2", "step_dispatch", "step_hll", "step_hllc", "step_fslp",
         "problems")


def build_with_fake_runtime(tmp_path, harness):
    """The executable, or None where it cannot be built."""
    from fv2d_gb300 import build as b
    cxx = shutil.which(os.environ.get("CXX", "g++")) or shutil.which("g++")
    try:
        nvcc = b._nvcc()
    except RuntimeError:
        return None
    roots = [os.environ.get("CUDA_HOME", ""), *(os.path.dirname(os.path.dirname(f(nvcc)))
                                                for f in (os.path.abspath, os.path.realpath)), "/usr/local/cuda"]
    include = next((d for r in roots for d in [os.path.join(r, "include"),
                                               *glob.glob(os.path.join(r, "targets", "*", "include"))]
                    if os.path.exists(os.path.join(d, "cuda_runtime_api.h"))), None)
    if not cxx or not include:
        return None
    b.build()
    exe = str(tmp_path / "harness")
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I" + include, "-o", exe,
                    os.path.join(REPO, "tests", harness)] + [os.path.join(b.BUILD, u + ".o") for u in UNITS],
                   check=True)
    return exe
