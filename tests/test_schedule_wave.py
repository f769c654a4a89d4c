"""The full-wave band height of the service's march lanes, on the host against a
restatement: the shortest of 1..18 rows whose work items fit the resident
warps, else of 8..16 rows whose items fit them twice over, else 0."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from fv2d_testlib import REPO


def rule(grids, warps):
    for waves, heights in ((1, range(1, 19)), (2, range(8, 17))):
        for H in heights:
            if sum(s * -(-ny // H) for s, ny in grids) <= waves * warps:
                return H
    return 0


def test_wave_band_matches_the_rule(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++")) or shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "wave")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-o", exe,
                    os.path.join(REPO, "tests", "schedule_wave_harness.cpp")], check=True)
    rng = np.random.default_rng(3)
    # lone grids: 128^2 a row an item, 512^2 two, RT 512 x 1536 ten, 2048^2 two waves of 15, 4096^2 none
    cases = [([(3, 128)], 2432.0), ([(9, 512)], 2432.0), ([(19, 1536)], 3040.0), ([(35, 2048)], 2432.0),
             ([(69, 4096)], 2432.0), ([(1, 18)], 1.0), ([(1, 19)], 1.0), ([(1, 33)], 1.0)]
    expect = [1, 2, 10, 15, 0, 18, 10, 0]
    for _ in range(300):
        n = int(rng.integers(1, 30))
        cases.append(([(int(rng.integers(1, 40)), int(rng.integers(16, 1500))) for _ in range(n)],
                      float(rng.choice([2432.0, 3040.0, 1216.0]))))
    text = "".join(f"{len(g)} {w!r}\n" + "".join(f"{s} {ny}\n" for s, ny in g) for g, w in cases)
    r = subprocess.run([exe], input=text, capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    got = [int(x) for x in r.stdout.split()]
    assert got[:len(expect)] == expect
    for (grids, warps), h in zip(cases, got):
        assert h == rule(grids, warps), (grids, warps)
