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
