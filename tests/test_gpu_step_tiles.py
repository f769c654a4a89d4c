"""The FP64 step's tile choice at its edges, bit for bit against the oracle:
grids on both sides of the small-tile limit (456 tiles of 8 x 8) and grids that
cut tiles."""
import numpy as np
import pytest

from fv2d_testlib import Oracle, bits_equal, reference_params

pytestmark = pytest.mark.gpu

RNG = np.random.default_rng(17)


def state(kind, nx, ny):
    q = np.empty((ny, nx, 4))
    q[..., 0] = 1.0 + 0.3 * RNG.random((ny, nx))
    q[..., 1:3] = 0.4 * RNG.random((ny, nx, 2)) - 0.2
    q[..., 3] = 1.0 + 0.3 * RNG.random((ny, nx))
    return q


@pytest.mark.parametrize("nx,ny", [(152 * 8, 24), (152 * 8 + 1, 24), (5, 3), (17, 9), (33, 70), (8, 8), (16, 16),
                                   (300, 301)])
@pytest.mark.parametrize("recon,solver", [(2, 1), (3, 0), (0, 2)])
def test_tile_edges_match_oracle(gpu_lib, nx, ny, recon, solver):
    import fv2d_gb300 as fv
    p = reference_params(Nx=nx, Ny=ny, gamma0=1.4, CFL=0.5, reconstruction=recon, riemann_solver=solver,
                         boundary_x=nx % 3, boundary_y=ny % 3, time_stepping=nx % 2)
    q = state("random", nx, ny)
    o, s = Oracle(p), fv.Simulation(p)
    o.set_prim(q)
    s.set_prim(q)
    for _ in range(3):
        d = o.compute_dt()[0]
        assert bits_equal(s.compute_dt()[0], d)
        o.update(d)
        s.update(d)
    assert bits_equal(s.get_prim(), o.get_prim())
