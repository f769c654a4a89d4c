"""Requests admitted and retired together: their conservation sums (one launch
for up to 64 of them) and final states, against sums of the state the service
returns.  Sizes from less than one CTA's cells to many CTAs', more requests
than one launch takes, rows that do not divide by a warp's 128 words."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(16, 16)] * 70 + [(300, 500)], [(1030, 700), (129, 33), (17, 2000)]])
def test_sums_match_the_returned_states(gpu_lib, sizes):
    import fv2d_gb300 as fv
    from fv2d_gb300.serve import Server
    with Server(budget_bytes=4e9, autotune=False) as s:
        reqs = []
        for k, (nx, ny) in enumerate(sizes):
            p = fv.default_params(Nx=nx, Ny=ny, gamma0=fv.as_float32(1.4), CFL=0.5, reconstruction=fv.PLM,
                                  boundary_x=fv.BC_PERIODIC, boundary_y=fv.BC_PERIODIC, seed=k + 1)
            # max_steps 0: retired as admitted, both sums are of the initial state
            reqs.append((s.submit("kh_step", p, 3 if k % 2 else 0), p))
        assert s.drain(60) == 0
        res = {r.id: r for r in s.poll()}
        for rid, p in reqs:
            r, q = res[rid], s.get_prim(rid)
            assert r.status == 0
            area = ((p.xmax - p.xmin) / p.Nx) * ((p.ymax - p.ymin) / p.Ny)
            rho, u, v, prs = (q[..., k] for k in range(4))
            cons = [rho, rho * u, rho * v, 0.5 * rho * (u * u + v * v) + prs / (p.gamma0 - 1.0)]
            # the recovered state is a few binary64 roundings from the summed
            # one, per cell and per partial sum: 1e-13 of the sum of magnitudes
            for k in range(4):
                assert abs(r.cons1[k] - cons[k].sum() * area) <= 1e-13 * np.abs(cons[k]).sum() * area
            if r.steps == 0:
                assert list(r.cons0) == list(r.cons1)
            s.release(rid)
