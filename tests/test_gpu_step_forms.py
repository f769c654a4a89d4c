"""The FP64 step's instantiations (plain Euler steps; with sources or RK2
stages) and its ghost cells, bit for bit against the oracle."""
import numpy as np
import pytest

from fv2d_testlib import Oracle, bits_equal, reference_params

pytestmark = pytest.mark.gpu

FORMS = {"plain": {}, "rk2": dict(time_stepping=1), "gravity": dict(gravity_mode=1, gx=0.1, gy=-0.2),
         "well-balanced": dict(gravity_mode=1, gy=-0.2, well_balanced_flux_at_y_bc=1),
         "conduction": dict(thermal_conductivity_active=1, kappa=1e-3)}


def check(p, nx, ny):
    import fv2d_gb300 as fv
    rng = np.random.default_rng(nx * 100 + ny)
    q = np.empty((ny, nx, 4))
    q[..., 0] = 1.0 + 0.3 * rng.random((ny, nx))
    q[..., 1:3] = 0.4 * rng.random((ny, nx, 2)) - 0.2
    q[..., 3] = 1.0 + 0.3 * rng.random((ny, nx))
    o, s = Oracle(p), fv.Simulation(p)
    o.set_prim(q)
    s.set_prim(q)
    for _ in range(3):
        d = o.compute_dt()[0]
        assert bits_equal(s.compute_dt()[0], d)
        o.update(d)
        s.update(d)
    assert bits_equal(s.get_prim(), o.get_prim())


@pytest.mark.parametrize("nx,ny", [(19, 13), (152 * 8 + 1, 24)])  # small tiles, full tiles
@pytest.mark.parametrize("recon", [0, 2, 3])
@pytest.mark.parametrize("solver", [0, 1, 2])
@pytest.mark.parametrize("form", FORMS)
def test_every_form_matches_oracle(gpu_lib, form, solver, recon, nx, ny):
    check(reference_params(Nx=nx, Ny=ny, gamma0=1.4, CFL=0.5, reconstruction=recon, riemann_solver=solver,
                           boundary_x=1, boundary_y=1, **FORMS[form]), nx, ny)


@pytest.mark.parametrize("nx,ny", [(2, 2), (3, 2), (2, 5), (4, 4), (8, 9), (152 * 8 + 1, 24)])
@pytest.mark.parametrize("bcx", [0, 1, 2])
@pytest.mark.parametrize("bcy", [0, 1, 2])
def test_ghost_cells_of_narrow_grids(gpu_lib, nx, ny, bcx, bcy):
    """Narrow grids, where one cell has ghosts on both sides."""
    check(reference_params(Nx=nx, Ny=ny, gamma0=1.4, CFL=0.5, reconstruction=2, riemann_solver=1, boundary_x=bcx,
                           boundary_y=bcy), nx, ny)
