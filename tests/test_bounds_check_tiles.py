"""The bounds-check build (-DFV2D_BOUNDS_CHECK) on grids of more than 456 tiles of
8 x 8 cells, which the FP64 step cuts into its 16 x 16 tiles (ragged ones, down
to two cells along an axis), and on the device loops of both tiles, where steps
commit each other and overlap: no index out of range, and per-step calls and
loops give the oracle's bits in both builds.  Every solver, reconstruction and
form of the step (plain, with sources, viscous; Euler and RK2)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from fv2d_testlib import Oracle, bits_equal, random_prim, reference_params

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
WIDE = [(24, 1217), (1217, 24), (175, 173), (2, 3700), (3700, 2), (171, 350)]
SMALL = [(13, 19), (2, 9), (64, 33)]
VISCOUS = dict(viscosity_active=1, mu=1e-2)
FORMS = [{}, dict(time_stepping=1),
         dict(gravity_mode=1, gx=0.05, gy=-0.1, well_balanced_flux_at_y_bc=1, thermal_conductivity_active=1,
              kappa=0.01), VISCOUS,
         dict(time_stepping=1, gravity_mode=1, gy=-0.1, thermal_conductivity_active=1, kappa=0.01, **VISCOUS)]
UPDATES, ADVANCED, QUEUED = 2, 5, 3


def cases():
    out = []
    for solver in (0, 1, 2):
        for recon in (0, 2, 3):
            for form in FORMS:
                k = len(out)
                shape = SMALL[k % 3] if k % 4 == 3 else WIDE[k % len(WIDE)]
                out.append((dict(riemann_solver=solver, reconstruction=recon, boundary_x=k % 3,
                                 boundary_y=(k // 3) % 3, **form), *shape))
    return out


def params(c, ny, nx):
    return reference_params(Nx=nx, Ny=ny, gamma0=1.4, CFL=0.4, **c)


def run(q0s, lib_path=None):
    """Per-step calls, a loop that stops at a step count, one that does not wait."""
    import fv2d_gb300 as fv
    if lib_path:
        fv.LIB_PATH = lib_path
    res, errs = [], []
    for case, q0 in zip(cases(), q0s):
        s = fv.Simulation(params(*case))
        s.set_prim(q0)
        for _ in range(UPDATES):
            s.update(s.compute_dt()[0])
        s.advance(ADVANCED, 1e30)
        s.run_async(QUEUED)
        res.append(s.get_prim())
        errs.append(s.device_errors())
        s.close()
    return res, errs


def test_tiles_and_loops_stay_in_bounds(gpu_lib, tmp_path):
    from fv2d_gb300 import build as b
    checked = b.build(bounds_check=True)
    q0s = [random_prim(ny, nx, 57 + k) for k, (_, ny, nx) in enumerate(cases())]
    np.savez(tmp_path / "in.npz", *q0s)
    script = f"""
import sys, numpy as np
sys.path[:0] = [{os.path.dirname(HERE)!r}, {HERE!r}]
from test_bounds_check_tiles import run
d = np.load({str(tmp_path / "in.npz")!r})
res, errs = run([d["arr_%d" % k] for k in range(len(d.files))], {checked!r})
np.savez({str(tmp_path / "out.npz")!r}, errs=np.array(errs), *res)
"""
    r = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    out = np.load(tmp_path / "out.npz")
    assert not out["errs"].any(), out["errs"]
    ref, errs = run(q0s)
    assert not any(errs)
    for k, (case, q0) in enumerate(zip(cases(), q0s)):
        o = Oracle(params(*case))
        o.set_prim(q0)
        for _ in range(UPDATES + ADVANCED + QUEUED):
            o.update(o.compute_dt()[0])
        assert bits_equal(ref[k], o.get_prim()), case
        assert bits_equal(out["arr_%d" % k], ref[k]), case
