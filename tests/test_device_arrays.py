"""The caller's arrays of set_prim_device and get_prim_device: which of them a
kernel uses itself (on the host, with a runtime that runs no kernels), and arrays
at odd addresses on the device."""
import subprocess

import pytest

from fake_runtime import build_with_fake_runtime
from fv2d_testlib import bits_equal, random_prim, reference_params


def test_other_arrays_are_staged(tmp_path):
    exe = build_with_fake_runtime(tmp_path, "device_array_harness.cpp")
    if not exe:
        pytest.skip("no C++ compiler or no built objects")
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 4, 8, 12, 16])  # bytes past a 256-byte boundary
def test_arrays_at_any_address(gpu_lib, offset):
    import torch
    import fv2d_gb300 as fv
    q = random_prim(33, 47, 5)
    s = fv.Simulation(reference_params(Nx=47, Ny=33, gamma0=1.4, CFL=0.5))
    pad = torch.zeros(q.nbytes + 512, dtype=torch.uint8, device="cuda")
    raw = pad[offset + (-pad.data_ptr()) % 256:][:q.nbytes]
    raw.copy_(torch.from_numpy(q.view("uint8").reshape(-1).copy()))
    torch.cuda.synchronize()
    s.set_prim_device(raw.data_ptr())
    assert bits_equal(s.get_prim(), q)
    raw.zero_()
    torch.cuda.synchronize()
    s.get_prim_device(raw.data_ptr())
    assert bits_equal(raw.cpu().numpy().view("float64").reshape(q.shape), q)
