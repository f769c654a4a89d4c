"""The service's guards in every register-resident step kernel: cells that a
step leaves with a negative density or pressure are counted, cells that it
leaves NaN fail the request (SimInfo.h:602-646)."""
import pytest

from fv2d_testlib import Oracle

pytestmark = pytest.mark.gpu

CONFIGS = ["28/32x20/march", "60/32x16/march2", "60/32x10/march2-diff"]
# problem, grid, CFL far above the stable one: (rho, p) resets of the first step
OVERSTEPS = [("sod_x", 61, 17, 4, "HLLC", (17, 0)), ("sod_x", 61, 17, 3, "HLLC", (0, 17)),
             ("sod_x", 61, 17, 3, "HLL", (17, 0)), ("blast", 61, 43, 3, "HLLC", (0, 28)),
             ("blast", 130, 43, 3, "HLL", None)]


def params(problem, nx, ny, cfl, solver, diffusive):
    import fv2d_gb300 as fv
    f = fv.as_float32
    walls = (fv.BC_ABSORBING, fv.BC_PERIODIC) if problem == "sod_x" else (fv.BC_REFLECTING, fv.BC_REFLECTING)
    extra = dict(thermal_conductivity_active=1, kappa=f(1e-6), viscosity_active=1, mu=f(1e-6)) if diffusive else {}
    return fv.default_params(Nx=nx, Ny=ny, gamma0=f(1.4), CFL=f(cfl), reconstruction=fv.PLM,
                             riemann_solver=getattr(fv, solver), boundary_x=walls[0], boundary_y=walls[1], **extra)


@pytest.mark.parametrize("lowmach", [False, True])
@pytest.mark.parametrize("diffusive", [False, True])
@pytest.mark.parametrize("config", CONFIGS)
def test_negative_cells_are_counted(gpu_lib, config, diffusive, lowmach):
    """One step past the stable one: the counts of the binary64 oracle.  The
    values of these states are of order 0.01 or more away from zero, a binary32
    step's rounding of order 1e-6, so the counts are equal."""
    from fv2d_gb300.serve import Server
    with Server(budget_bytes=1e9, autotune=False, tile_config=config) as s:
        ids, want = [], []
        for problem, nx, ny, cfl, solver, expected in OVERSTEPS:
            p = params(problem, nx, ny, cfl, solver, diffusive)
            o = Oracle(p)
            o.init_problem(problem)
            o.update(o.compute_dt()[0])
            c = o.counters()
            assert c[0] + c[1] > 0 and c[2] == 0
            if expected is not None:
                assert tuple(c[:2]) == expected
            ids.append(s.submit(problem, p, 1, lowmach=lowmach))
            want.append(c[0] + c[1])
        assert s.drain(120) == 0
        res = {r.id: r for r in s.poll()}
        assert [res[i].status for i in ids] == [0] * len(ids)
        assert [res[i].negatives for i in ids] == want


@pytest.mark.parametrize("diffusive", [False, True])
@pytest.mark.parametrize("stepping", ["TS_EULER", "TS_RK2"])
@pytest.mark.parametrize("config", CONFIGS)
def test_nan_cells_fail_their_request(gpu_lib, config, stepping, diffusive):
    import fv2d_gb300 as fv
    from fv2d_gb300._abi import ERR_NUMERIC
    from fv2d_gb300.serve import Server
    good = params("sod_x", 61, 17, 0.8, "HLLC", diffusive)
    bad = params("sod_x", 129, 17, 0.8, "HLLC", diffusive)
    for p in (good, bad):
        p.time_stepping = getattr(fv, stepping)
    bad.sod_rho_right = float("nan")
    with Server(budget_bytes=1e9, autotune=False, tile_config=config) as s:
        b, g = s.submit("sod_x", bad, 20), s.submit("sod_x", good, 20)
        assert s.drain(120) == 0
        res = {r.id: r for r in s.poll()}
        assert res[b].status == ERR_NUMERIC and res[b].steps < 20
        assert res[g].status == 0 and res[g].steps == 20


@pytest.mark.parametrize("scheme", ["plain", "diffusive", "extended"])
@pytest.mark.parametrize("bcx", ["BC_ABSORBING", "BC_REFLECTING", "BC_PERIODIC"])
def test_ghost_columns_of_any_width(gpu_lib, scheme, bcx):
    """The ghost cells that the march kernels write, at widths around their
    strips (28 and 60 columns) and at the narrowest grid, against the binary64
    path.  A step rounds each of its ~50 chained operations to 2^-24 of the
    fields' scale, so 8 steps stay below 8 * 50 * 6e-8 = 2.4e-5 of it; a wrong
    ghost is an error of order 0.01 in the cells beside it."""
    import numpy as np
    import fv2d_gb300 as fv
    from fv2d_gb300.serve import Server
    f = fv.as_float32
    extra = {"plain": {}, "diffusive": dict(thermal_conductivity_active=1, kappa=f(1e-4), viscosity_active=1,
                                            mu=f(1e-4)),
             "extended": dict(reconstruction=fv.MUSCL_HANCOCK)}[scheme]
    configs = {"plain": ["28/32x20/march", "60/32x16/march2"],
               "diffusive": ["28/32x20/march", "60/32x10/march2-diff"], "extended": [None]}[scheme]
    runs = []
    for nx in (16, 17, 27, 28, 29, 59, 60, 61, 62, 120, 121):
        for bcy, ny, ts in ((fv.BC_REFLECTING, 16, fv.TS_EULER), (fv.BC_PERIODIC, 19, fv.TS_RK2),
                            (fv.BC_ABSORBING, 21, fv.TS_EULER)):
            p = dict(Nx=nx, Ny=ny, gamma0=f(1.4), CFL=f(0.4), reconstruction=fv.PLM, riemann_solver=fv.HLLC,
                     boundary_x=getattr(fv, bcx), boundary_y=bcy, time_stepping=ts, seed=nx)
            p.update(extra)
            runs.append(fv.default_params(**p))
    for config in configs:
        with Server(budget_bytes=1e9, autotune=False, tile_config=config) as s:
            ids = [s.submit("kh_step", p, 8) for p in runs]
            assert s.drain(120) == 0
            res = {r.id: r for r in s.poll()}
            for p, i in zip(runs, ids):
                assert res[i].status == 0
                sim = fv.Simulation(p)
                sim.init_problem("kh_step")
                sim.advance(8, 1e30)
                want, got = np.asarray(sim.get_prim()), np.asarray(s.get_prim(i), dtype=float)
                scale = np.abs(want).max(axis=(0, 1))
                scale[1:3] = scale[1:3].max()
                assert (np.abs(got - want).max(axis=(0, 1)) <= 2.4e-5 * scale).all(), (config, p.Nx, p.Ny)
