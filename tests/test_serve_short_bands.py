"""The 2- to 7-row bands that full-wave lanes choose (band_rows cannot ask for
them), in every march kernel: the same bits as with bands of 8 and 13 rows."""
import pytest

from fv2d_testlib import bits_equal
from test_schedule_wave import rule

pytestmark = pytest.mark.gpu

SMS = 152
# kernel, its strip's columns, resident warps an SM, its requests' physics
KERNELS = [("28/32x20/march", 28, 20, "plain"), ("60/32x16/march2", 60, 16, "plain"), ("60/32x10/march2-diff", 60, 10, "diff"),
           ("28/64x8/march-ext", 28, 16, "mh")]
HEIGHTS = range(2, 8)


def grid(strip, warps, rows, odd):
    """A grid whose lane takes `rows`-row bands."""
    nx = 8 * strip - odd
    ny = (warps // 8) * rows - odd
    assert rule([(8, ny)], warps) == rows
    return nx, ny


@pytest.mark.parametrize("tile,strip,per_sm,physics", KERNELS)
def test_short_bands_leave_the_bits(gpu_lib, tile, strip, per_sm, physics):
    import torch
    import fv2d_gb300 as fv
    from fv2d_gb300.serve import Server
    if torch.cuda.get_device_properties(0).multi_processor_count != SMS:
        pytest.skip("the band heights below are a 152-SM device's")
    f = fv.as_float32
    extra = {"diff": dict(thermal_conductivity_active=1, kappa=f(1e-4), viscosity_active=1, mu=f(1e-4)),
             "mh": dict(reconstruction=fv.MUSCL_HANCOCK)}.get(physics, {})
    runs = []
    for k, rows in enumerate(HEIGHTS):
        nx, ny = grid(strip, SMS * per_sm, rows, k % 3)
        p = dict(Nx=nx, Ny=ny, gamma0=f(1.4), CFL=f(0.4), reconstruction=fv.PLM, riemann_solver=k % 2,
                 boundary_x=k % 3, boundary_y=(k + 1) % 3, time_stepping=k // 3, seed=k + 1)
        p.update(extra)
        runs.append(fv.default_params(**p))
    results = []
    for band in (0, 8, 13):
        with Server(budget_bytes=4e9, autotune=False, tile_config=tile, band_rows=band) as s:
            out = []
            for p in runs:  # one at a time: the lane holds this grid alone
                i = s.submit("kh_step", p, 4)
                assert s.drain(60) == 0
                r = s.poll()[0]
                assert r.status == 0 and r.steps == 4
                out.append((s.get_prim(i), r.t))
                s.release(i)
            results.append(out)
    for other in results[1:]:
        for p, (q, t), (q0, t0) in zip(runs, other, results[0]):
            assert t == t0 and bits_equal(q, q0), (p.Nx, p.Ny)
