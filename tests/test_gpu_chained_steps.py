"""Device-driven runs whose steps commit each other (grids of up to 2048 CTAs)
against per-step calls, bit for bit: run lengths around the replayed graph's 32
steps, ends inside it (step cap, end time, snapshot time), both schemes, both
tiles, overlapped and plain launches, the log and the counters; and a run that
goes on after another."""
import numpy as np
import pytest

from fv2d_testlib import bits_equal, reference_params

pytestmark = pytest.mark.gpu


def pair(nx, ny, ts):
    import fv2d_gb300 as fv
    p = reference_params(Nx=nx, Ny=ny, gamma0=1.4, CFL=0.5, reconstruction=2, riemann_solver=1, boundary_x=2,
                         boundary_y=1, time_stepping=ts)
    rng = np.random.default_rng(nx + ny)
    q = np.empty((ny, nx, 4))
    q[..., 0] = 1.0 + 0.3 * rng.random((ny, nx))
    q[..., 1:3] = 0.4 * rng.random((ny, nx, 2)) - 0.2
    q[..., 3] = 1.0 + 0.3 * rng.random((ny, nx))
    sims = fv.Simulation(p), fv.Simulation(p)
    for s in sims:
        s.set_prim(q)
    return sims


# 32 small tiles; 400 small (no overlap); 196 wide (no overlap); 500 wide (overlap); 2116 wide (not chained)
@pytest.mark.parametrize("nx,ny", [(64, 32), (160, 160), (224, 224), (400, 320), (736, 736)])
@pytest.mark.parametrize("ts", [0, 1])
def test_driven_runs_match_single_steps(gpu_lib, nx, ny, ts):
    a, b = pair(nx, ny, ts)
    done = 0
    for n in (1, 5, 33) if nx < 700 else (1, 5):
        t, steps, status = a.advance(n, 1e30)
        assert (steps, status) == (n, 0)
        log = a.step_log()
        assert len(log) == n
        for k in range(n):
            dt, hyp, _, _ = b.compute_dt()
            assert bits_equal(log[k, 1:3], np.array([dt, hyp])) and log[k, 0] == b.time()[0]
            b.update(dt)
        done += n
        assert a.time() == b.time() and a.time()[1] == done
        assert bits_equal(a.compute_dt()[0], b.compute_dt()[0])
        assert bits_equal(a.get_prim(), b.get_prim())
        assert a.counters() == b.counters()
    a.run_async(3)
    for _ in range(3):
        b.update(b.compute_dt()[0])
    assert bits_equal(a.get_prim(), b.get_prim()) and a.time() == b.time()


@pytest.mark.parametrize("nx,ny", [(64, 32), (400, 320)])
def test_runs_stop_inside_a_replay(gpu_lib, nx, ny):
    import fv2d_gb300 as fv
    a, b = pair(nx, ny, 0)
    for _ in range(7):
        b.update(b.compute_dt()[0])
    t7 = b.time()[0]
    eps = a.params.epsilon
    # a snapshot due within epsilon after step 7, then the end of the run there
    t, n, status = a.advance(1000, 1e30, next_save=t7 + eps / 2)
    assert (n, status, t) == (7, fv.RUN_SAVE, t7) and bits_equal(a.get_prim(), b.get_prim())
    t, n, status = a.advance(1000, t7 + eps / 2)
    assert (n, status, t) == (0, fv.RUN_DONE, t7) and bits_equal(a.get_prim(), b.get_prim())
    a.update(a.compute_dt()[0])
    b.update(b.compute_dt()[0])
    assert bits_equal(a.get_prim(), b.get_prim()) and a.time() == b.time()
