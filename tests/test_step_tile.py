"""The FP64 step's tile and overlapped launches by the device's SM count, on the
host: 8 x 8 tiles while they are at most three to an SM, and overlap at up to two
small tiles an SM or more than three wide ones (up to 2048 of them)."""
import subprocess

import pytest

from fake_runtime import build_with_fake_runtime


def rule(sms, nx, ny):
    small, wide = -(-nx // 8) * -(-ny // 8), -(-nx // 16) * -(-ny // 16)
    if small <= 3 * sms:
        return 8, int(small <= 2 * sms)
    return 16, int(3 * sms < wide <= 2048)


def test_tile_and_overlap_follow_the_sm_count(tmp_path):
    exe = build_with_fake_runtime(tmp_path, "step_tile_harness.cpp")
    if not exe:
        pytest.skip("no C++ compiler or no built objects")
    grids = [(8 * 152, 16), (8 * 152 + 1, 16), (8 * 152, 24), (8 * 152 + 1, 24), (16 * 152, 48), (16 * 152 + 1, 48),
             (512, 1024), (528, 1024), (2, 2), (160, 160), (304, 16), (305, 24)]
    cases = [(sms, nx, ny) for sms in (152, 148, 76, 1) for nx, ny in grids]
    r = subprocess.run([exe], input="".join("%d %d %d\n" % c for c in cases), capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, r.stderr
    got = [tuple(map(int, line.split())) for line in r.stdout.split("\n") if line]
    assert got == [rule(*c) for c in cases]
