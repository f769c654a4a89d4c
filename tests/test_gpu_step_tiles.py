"""The FP64 step's tile choice and its dt reduction at their edges, bit for bit
against the oracle: grids on both sides of the small-tile limit (456 tiles of
8 x 8), grids that cut tiles, and states whose largest inverse dt sits where
the reduction's binary32 bound is tight, tied or does not apply."""
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
    if kind == "uniform":  # every cell ties
        q[:] = (1.0, 0.25, -0.125, 0.7)
    elif kind == "last":  # the maximum is one cell, by less than a binary32 ulp
        q[:] = (1.0, 0.25, -0.125, 0.7)
        q[-1, -1, 3] *= 1.0 + 1e-9
    elif kind == "small":  # sound speeds below the bound's range
        q[..., 1:3] *= 1e-30
        q[..., 3] *= 1e-60
    elif kind == "large":  # outside binary32
        q[..., 3] *= 1e90
    elif kind == "mixed":
        q[0, 0, 3] *= 1e60
        q[-1, 0, 3] *= 1e-60
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


@pytest.mark.parametrize("kind", ["random", "uniform", "last", "small", "large", "mixed"])
@pytest.mark.parametrize("nx,ny", [(40, 36), (400, 333)])
def test_dt_reduction_matches_oracle(gpu_lib, kind, nx, ny):
    import torch
    import fv2d_gb300 as fv
    p = reference_params(Nx=nx, Ny=ny, gamma0=1.4, CFL=0.5, reconstruction=2, boundary_x=2, boundary_y=2)
    q = state(kind, nx, ny)
    o, s = Oracle(p), fv.Simulation(p)
    o.set_prim(q)
    s.set_prim(q)
    d = o.compute_dt()
    assert bits_equal(np.array(s.compute_dt()), np.array(d))  # the set-up pass
    for offset in (0, 1):  # a 16-byte aligned array, and one that is not
        buf = torch.empty(q.size + 2, dtype=torch.float64, device="cuda")
        dev = buf[offset:offset + q.size]
        dev.copy_(torch.from_numpy(q).reshape(-1))
        out = torch.empty(4, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert fv.compute_dt_noalloc(p, dev.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        assert bits_equal(out.cpu().numpy(), np.array(d))
    for _ in range(2):  # the step
        o.update(d[0])
        s.update(d[0])
        d = o.compute_dt()
        assert bits_equal(s.compute_dt()[0], d[0])
