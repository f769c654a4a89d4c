"""The workloads this framework is timed on: the binary64 step loop, the
per-step calls of a host program, the allocation-free dt, and the batched
binary32 service, each through the calls a user's program makes.

A case is a dict of plain values:
  kind      "loop"   set_prim_device, a device-driven run, get_prim_device
            "host"   set_prim, (compute_dt, update) per step, get_prim, host arrays
            "dt"     compute_dt_noalloc of a device array
            "served" requests submitted to a running Server, drained and read back
  nx, ny    grid (the largest one of a "served" batch)
  problem   initial condition (seeded: see initial_values)
  recon, solver, ts, physics, bcx, bcy
            the scheme, the source and diffusion terms, the boundaries
  steps     time steps of one pass (of the longest request of a batch)
  count     requests of a batch
"""
import math
import random

import numpy as np
import torch

import fv2d_gb300 as fv
from fv2d_gb300._abi import OK
from fv2d_gb300.serve import Server

RECON = {"pcm": fv.PCM, "plm": fv.PLM, "mh": fv.MUSCL_HANCOCK}
SOLVER = {"hll": fv.HLL, "hllc": fv.HLLC, "fslp": fv.FSLP}
STEPPING = {"euler": fv.TS_EULER, "rk2": fv.TS_RK2}
BOUNDARY = {"absorbing": fv.BC_ABSORBING, "reflecting": fv.BC_REFLECTING, "periodic": fv.BC_PERIODIC}
# x and y boundaries each problem is run with
WALLS = {"sod_x": ("absorbing", "periodic"), "blast": ("reflecting", "reflecting"),
         "sedov": ("reflecting", "reflecting"), "kh_step": ("periodic", "periodic"),
         "gresho_vortex": ("periodic", "periodic"), "rt_hydrostatic": ("periodic", "reflecting")}
# gravity, conduction and viscosity of the Rayleigh-Taylor set-up
PHYSICS = {"none": {},
           "gravity": dict(gravity_mode=fv.GRAV_CONSTANT, gy=-0.1),
           "diffusive": dict(gravity_mode=fv.GRAV_CONSTANT, gy=-0.1, thermal_conductivity_active=1, kappa=1e-4,
                             viscosity_active=1, mu=1e-4)}
SERVED_PLAIN = ("sod_x", "sedov", "kh_step", "gresho_vortex")
MOST_CELL_STEPS = 4 * 4096 * 4096  # of a binary64 case
MOST_SERVED_CELL_STEPS = 200 * 2048 * 2048


def _case(kind, nx, ny, problem, recon="plm", solver="hllc", ts="euler", physics="none", steps=1, count=1, **more):
    return dict(kind=kind, nx=nx, ny=ny, problem=problem, recon=recon, solver=solver, ts=ts, physics=physics,
                steps=steps, count=count, **more)


def listed():
    return [
        # the 1-D Sod tube of the CPU benchmark (MUSCL-Hancock, HLLC): the smallest grids, where a step is latency
        _case("loop", 512, 8, "sod_x", recon="mh", steps=100, call="advance", name="sod 512x8"),
        # the reference's blast settings grid, advanced on the device between two snapshots
        _case("loop", 256, 256, "blast", steps=64, call="advance", name="blast 256"),
        # the headline benchmark
        _case("loop", 2048, 2048, "sedov", steps=16, call="run_async", name="sedov 2048"),
        # the largest benchmark grid: every cell in motion
        _case("loop", 4096, 4096, "kh_step", steps=4, call="run_async", name="kh 4096"),
        # the Rayleigh-Taylor benchmark: HLL, gravity, conduction and viscosity
        _case("loop", 1024, 3072, "rt_hydrostatic", solver="hll", physics="diffusive", steps=8, call="run_async",
              name="rt 1024x3072"),
        # a ragged grid with the two-stage scheme and the low-Mach solver
        _case("loop", 777, 1501, "rt_hydrostatic", solver="fslp", ts="rk2", physics="gravity", steps=8,
              call="run_async", name="fslp rk2 777x1501"),
        # a host program that swaps its own update and dt calls for the library's, host arrays in and out
        _case("host", 1000, 600, "kh_step", solver="hll", recon="pcm", steps=5, name="host steps 1000x600"),
        # the dt of an array some other allocator owns
        _case("dt", 3000, 2000, "kh_step", name="dt 3000x2000"),
        # one large request, read back when done
        _case("served", 2048, 2048, "kh_step", steps=200, name="served kh 2048"),
        # a burst of the request stream: grids of 64 to 512 cells a side, four problems
        _case("served", 512, 512, "mix", steps=200, count=16, name="served mix"),
        # the diffusive kernel family
        _case("served", 512, 1536, "rt_hydrostatic", solver="hll", physics="diffusive", steps=200,
              name="served rt 512x1536"),
        # the extended kernel family: MUSCL-Hancock and FSLP, Euler and RK2, odd rectangles
        _case("served", 320, 480, "extended", steps=80, count=6, name="served extended"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop"] * 5 + ["host", "dt"] + ["served"] * 3)
    if kind == "dt":
        return _case("dt", _log_int(rng, 64, 4096), _log_int(rng, 64, 4096), "kh_step")
    if kind == "served":
        form = rng.choice(["one", "mix", "rt", "extended"])
        if form == "mix":
            return _case("served", 512, 512, "mix", steps=rng.randint(100, 200), count=rng.randint(4, 16))
        if form == "extended":
            return _case("served", rng.randint(64, 320), rng.randint(64, 480), "extended",
                         steps=rng.randint(40, 80), count=rng.randint(2, 6))
        nx, ny = _log_int(rng, 64, 2048), _log_int(rng, 64, 2048)
        steps = max(100, min(200, MOST_SERVED_CELL_STEPS // (nx * ny)))
        if form == "rt":
            return _case("served", nx, ny, "rt_hydrostatic", solver="hll", physics="diffusive", steps=steps)
        return _case("served", nx, ny, rng.choice(["sod_x", "sedov", "kh_step"]), steps=steps)
    problem = rng.choice(["sod_x", "blast", "sedov", "kh_step", "rt_hydrostatic"])
    solver = rng.choice(["hll", "hllc", "hllc", "fslp"])
    recon = rng.choice(["pcm", "plm", "plm", "mh"])
    ts = rng.choice(["euler", "euler", "rk2"])
    physics = rng.choice(["gravity", "diffusive"]) if problem == "rt_hydrostatic" else "none"
    if kind == "host":
        nx, ny = _log_int(rng, 64, 1200), _log_int(rng, 64, 1200)
        return _case("host", nx, ny, problem, recon, solver, ts, physics, rng.randint(1, 6))
    nx, ny = _log_int(rng, 64, 4096), _log_int(rng, 8, 4096)
    stages = 2 if ts == "rk2" else 1
    steps = max(1, min(100, MOST_CELL_STEPS // (2 * stages * nx * ny)))
    return _case("loop", nx, ny, problem, recon, solver, ts, physics, steps,
                 call="advance" if nx * ny < 1 << 18 else "run_async")


# ------------------------------------------------------------- set-ups
def _values(rng, problem):
    """The seeded physical values of one set-up (the ranges of the request stream)."""
    v = dict(problem=problem, gamma0=fv.as_float32(rng.uniform(1.3, 1.67)))
    if problem == "sod_x":
        v.update(sod_rho_left=1.0, sod_p_left=1.0, sod_rho_right=1.0 / rng.uniform(2.0, 20.0), sod_p_right=0.1)
    elif problem == "sedov":
        v.update(sedov_E0=rng.uniform(0.5, 2.0))
    elif problem == "kh_step":
        v.update(khs_u=rng.uniform(0.2, 1.0), khs_noise=0.0)
    elif problem == "gresho_vortex":
        v.update(gresho_density=1.0, gresho_Mach=fv.as_float32(rng.uniform(0.01, 0.1)))
    elif problem == "rt_hydrostatic":
        v.update(rt_amp=rng.uniform(0.005, 0.02))
    elif problem == "blast":
        v.update(blast_p=rng.uniform(5.0, 20.0))
    return v


def _domain(problem):
    return (0.5, 1.5) if problem == "rt_hydrostatic" else (1.0, 1.0)


def _params(nx, ny, v, recon, solver, ts, physics):
    xmax, ymax = _domain(v["problem"])
    bcx, bcy = WALLS[v["problem"]]
    if v["problem"] == "sod_x" and ny < nx // 4:
        ymax = ny / nx  # a tube of square cells
    p = fv.default_params(Nx=nx, Ny=ny, xmax=xmax, ymax=ymax, CFL=fv.as_float32(0.7), reconstruction=RECON[recon],
                          riemann_solver=SOLVER[solver], time_stepping=STEPPING[ts], boundary_x=BOUNDARY[bcx],
                          boundary_y=BOUNDARY[bcy], **PHYSICS[physics])
    return p.update(**{k: x for k, x in v.items() if k not in ("problem", "blast_p")})


def initial_values(p, v, device):
    """Interior primitives (4, Ny, Nx) of a problem in binary64."""
    dx, dy = (p.xmax - p.xmin) / p.Nx, (p.ymax - p.ymin) / p.Ny
    x = p.xmin + (torch.arange(p.Nx, device=device, dtype=torch.float64) + 0.5) * dx
    y = p.ymin + (torch.arange(p.Ny, device=device, dtype=torch.float64) + 0.5) * dy
    y, x = torch.meshgrid(y, x, indexing="ij")
    xr, yr = x - 0.5 * (p.xmin + p.xmax), y - 0.5 * (p.ymin + p.ymax)
    r = torch.sqrt(xr * xr + yr * yr)
    rho, u, vv, prs = torch.ones_like(x), torch.zeros_like(x), torch.zeros_like(x), torch.ones_like(x)
    problem = v["problem"]
    if problem == "sod_x":
        left = x <= 0.5
        rho = torch.where(left, p.sod_rho_left, p.sod_rho_right * rho)
        prs = torch.where(left, p.sod_p_left, p.sod_p_right * prs)
    elif problem == "blast":
        rho = torch.where(r < 0.2, rho, 1.2)
        prs = torch.where(r < 0.2, v["blast_p"] * prs, 0.1)
    elif problem == "sedov":
        inside = (p.gamma0 - 1.0) * p.sedov_E0 / (math.pi * p.sedov_r0 ** 2)
        rho = p.sedov_rho * rho
        prs = torch.where(r <= p.sedov_r0, inside * prs, p.sedov_p_ambient)
    elif problem == "kh_step":
        inside = yr.abs() < 0.25
        rho = torch.where(inside, p.khs_rho_in * rho, p.khs_rho_out)
        u = torch.where(inside, p.khs_u + u, -p.khs_u)
        vv = p.khs_amp * torch.sin(4.0 * math.pi * x)
        prs = p.khs_p0 * prs
    elif problem == "gresho_vortex":
        p0 = p.gresho_density / (p.gamma0 * p.gresho_Mach * p.gresho_Mach)
        near, mid = r < 0.2, r < 0.4
        u_phi = torch.where(near, 5.0 * r, torch.where(mid, 2.0 - 5.0 * r, 0.0 * r))
        ring = p0 + 12.5 * r * r + 4.0 * (1.0 - 5.0 * r + torch.log(5.0 * r))
        prs = torch.where(near, p0 + 12.5 * r * r, torch.where(mid, ring, p0 - 2.0 + 4.0 * math.log(2.0) + 0.0 * r))
        rho = p.gresho_density * rho
        u, vv = -yr / r * u_phi, xr / r * u_phi
    elif problem == "rt_hydrostatic":
        rho = torch.where(y > p.rt_y_interface, p.rt_rho_top * rho, p.rt_rho_bottom)
        above = y - p.rt_y_interface
        vv = p.rt_amp * (1.0 + torch.cos(4.0 * math.pi * x)) * (1.0 + torch.cos(3.0 * math.pi * above)) / 4.0
        prs = p.rt_p_interface + rho * p.gy * above
    return torch.stack([rho, u, vv, prs])


def _one(case, seed, device):
    """Parameters and initial primitives (Ny, Nx, 4) of a single binary64 run."""
    rng = random.Random(seed)
    v = _values(rng, case["problem"])
    p = _params(case["nx"], case["ny"], v, case["recon"], case["solver"], case["ts"], case["physics"])
    q = initial_values(p, v, device)
    if case["problem"] in ("kh_step", "rt_hydrostatic"):  # the seeded noise that breaks the set-up's symmetry
        g = torch.Generator(device=device).manual_seed(seed)
        noise = torch.rand((2, p.Ny, p.Nx), generator=g, device=device, dtype=torch.float64)
        q[1:3] += 1e-3 * (2.0 * noise - 1.0)
    return p, q.permute(1, 2, 0).contiguous()


def _requests(case, seed):
    """(values, params, steps) of every request of a served batch."""
    rng = random.Random(seed)
    shape = random.Random(case["nx"] * 7919 + case["steps"])  # sizes belong to the case, values to the seed
    out = []
    for k in range(case["count"]):
        nx, ny, steps = case["nx"], case["ny"], case["steps"]
        recon, solver, ts, physics, problem = (case[n] for n in ("recon", "solver", "ts", "physics", "problem"))
        if problem == "mix":
            n = nx if k == 0 else max(64, 32 * round(_log_int(shape, 64, nx) / 32))
            nx, ny, steps, problem = n, n, shape.randint(steps // 2, steps), SERVED_PLAIN[k % 4]
        elif problem == "extended":
            nx, ny = (nx, ny) if k == 0 else (_log_int(shape, 32, nx), _log_int(shape, 32, ny))
            recon, solver, ts, physics, problem = [
                ("mh", "hllc", "euler", "none", "sod_x"), ("plm", "fslp", "rk2", "gravity", "rt_hydrostatic"),
                ("mh", "hll", "rk2", "diffusive", "rt_hydrostatic"), ("pcm", "fslp", "euler", "none", "kh_step"),
            ][k % 4]
        v = _values(rng, problem)
        out.append((v, _params(nx, ny, v, recon, solver, ts, physics), steps))
    return out


_SERVER = []


def _server():
    """The service of this process: a program starts one and keeps it."""
    if not _SERVER:
        _SERVER.append(Server(budget_bytes=60e9))
    return _SERVER[0]


# ------------------------------------------------------------- the calls
def prepare(case, seed):
    if case["kind"] == "served":
        return dict(kind="served", server=_server(), requests=_requests(case, seed))
    p, q = _one(case, seed, "cuda")
    if case["kind"] == "dt":
        return dict(kind="dt", p=p, q=q)
    sim = fv.Simulation(p)
    state = dict(kind=case["kind"], sim=sim, q=q, steps=case["steps"], call=case.get("call"))
    if case["kind"] == "host":
        state["q"] = q.cpu().numpy()
    return state


def run(state):
    kind = state["kind"]
    if kind == "loop":
        sim, q = state["sim"], state["q"]
        out = torch.empty_like(q)
        sim.set_prim_device(q.data_ptr())
        if state["call"] == "advance":
            sim.advance(state["steps"], 1e30)
        else:
            sim.run_async(state["steps"])
        sim.get_prim_device(out.data_ptr())
        return dict(prim=out, dt=sim.compute_dt()[0])
    if kind == "host":
        sim = state["sim"]
        sim.set_prim(state["q"])
        for _ in range(state["steps"]):
            sim.update(sim.compute_dt()[0])
        return dict(prim=sim.get_prim(), dt=sim.compute_dt()[0])
    if kind == "dt":
        out = torch.empty(4, device="cuda", dtype=torch.float64)
        stream = torch.cuda.current_stream().cuda_stream
        if fv.compute_dt_noalloc(state["p"], state["q"].data_ptr(), out.data_ptr(), stream) != OK:
            raise RuntimeError("compute_dt_noalloc failed")
        return out
    server = state["server"]
    ids = [server.submit(v["problem"], p, steps, lowmach=v["problem"] == "gresho_vortex")
           for v, p, steps in state["requests"]]
    if server.drain() != OK:
        raise RuntimeError("the service did not finish: " + server.last_error())
    if any(r.status != OK for r in server.poll()):
        raise RuntimeError("a request failed")
    out = []
    for rid in ids:
        # the service's states are binary32: a program that keeps many of them keeps them as that
        out.append(torch.from_numpy(server.get_prim(rid)).to(torch.float32))
        server.release(rid)
    return out


def work(case):
    if case["kind"] == "dt":
        return dict(bytes=32.0 * case["nx"] * case["ny"], flops=12.0 * case["nx"] * case["ny"])
    # per cell and stage: the conservative state read once and written once; about 250 operations
    if case["kind"] == "served":
        cells = sum(p.Nx * p.Ny * steps * (2 if p.time_stepping == fv.TS_RK2 else 1)
                    for _, p, steps in _requests(case, 0))
        return dict(bytes=32.0 * cells, flops=250.0 * cells)
    cells = case["nx"] * case["ny"]
    stages = case["steps"] * (2 if case["ts"] == "rk2" else 1)
    return dict(bytes=64.0 * cells * (stages + 1), flops=250.0 * cells * stages)


# ------------------------------------------------------------- 64-bit reference (plain torch)
def _sources(n, bc, device):
    k = torch.arange(-2, n + 2, device=device)
    if bc == fv.BC_REFLECTING:
        src = torch.where(k < 0, -k - 1, torch.where(k >= n, 2 * n - k - 1, k))
    elif bc == fv.BC_PERIODIC:
        src = k % n
    else:
        src = k.clamp(0, n - 1)
    outside = (k < 0) | (k >= n)
    sign = torch.where(outside & (bc == fv.BC_REFLECTING), -1.0, 1.0).to(torch.float64)
    return src, sign


def _padded(q, p):
    sx, gx = _sources(p.Nx, p.boundary_x, q.device)
    sy, gy = _sources(p.Ny, p.boundary_y, q.device)
    q = q[:, sy][:, :, sx]
    q[1] *= gx
    q[2] *= gy[:, None]
    return q


def _minmod(a, b):
    return torch.where(a * b < 0, 0.0, torch.where(a.abs() < b.abs(), a, b))


def _cons(q, gm1):
    r, u, v, p = q
    return torch.stack([r, r * u, r * v, 0.5 * r * (u * u + v * v) + p / gm1])


def _prim(c, gm1):
    r, u, v = c[0], c[1] / c[0], c[2] / c[0]
    return torch.stack([r, u, v, (c[3] - 0.5 * r * (u * u + v * v)) * gm1])


def _flux(L, R, p, gd):
    g = p.gamma0
    (rL, uL, vL, pL), (rR, uR, vR, pR) = L, R
    cL, cR = torch.sqrt(g * pL / rL), torch.sqrt(g * pR / rR)
    if p.riemann_solver == fv.FSLP:
        a = p.fslp_K * torch.maximum(rL * cL, rR * cR)
        theta = torch.maximum(uL.abs() / cL, uR.abs() / cR).clamp(max=1.0)
        us = 0.5 * (uR + uL) - 0.5 / a * (pR - pL - 0.5 * (rL + rR) * gd)
        pi = 0.5 * (pR + pL) - 0.5 * theta * a * (uR - uL)
        r, u, v, q = torch.where(us > 0, L, R)
        e = 0.5 * r * (u * u + v * v) + q / (g - 1.0)
        return torch.stack([us * r, us * r * u + pi, us * r * v, us * (e + pi)])
    eL = 0.5 * rL * (uL * uL + vL * vL) + pL / (g - 1.0)
    eR = 0.5 * rR * (uR * uR + vR * vR) + pR / (g - 1.0)
    if p.riemann_solver == fv.HLL:
        sL, sR = torch.minimum(uL - cL, uR - cR), torch.maximum(uL + cL, uR + cR)
        fL = torch.stack([rL * uL, rL * uL * uL + pL, rL * uL * vL, (pL + eL) * uL])
        fR = torch.stack([rR * uR, rR * uR * uR + pR, rR * uR * vR, (pR + eR) * uR])
        wL, wR = torch.stack([rL, rL * uL, rL * vL, eL]), torch.stack([rR, rR * uR, rR * vR, eR])
        mid = (sR * fL - sL * fR + sL * sR * (wR - wL)) / (sR - sL)
        return torch.where(sL >= 0, fL, torch.where(sR <= 0, fR, mid))
    c = torch.maximum(cL, cR)
    sL, sR = torch.minimum(uL, uR) - c, torch.maximum(uL, uR) + c
    mL, mR = rL * (uL - sL), rR * (sR - uR)
    us = (mR * uR + mL * uL + (pL - pR)) / (mR + mL)
    ps = (mR * pL + mL * pR + mL * mR * (uL - uR)) / (mR + mL)
    left = us > 0
    r, u, v, q = torch.where(left, L, R)
    e, s = torch.where(left, eL, eR), torch.where(left, sL, sR)
    rs, es = r * (s - u) / (s - us), ((s - u) * e - q * u + ps * us) / (s - us)
    star = torch.stack([rs, us, v, ps, es])
    wL, wR = torch.stack([rL, uL, vL, pL, eL]), torch.stack([rR, uR, vR, pR, eR])
    r, u, v, q, e = torch.where(sL > 0, wL, torch.where(left | (sR > 0), star, wR))
    return torch.stack([r * u, r * u * u + q, r * u * v, (e + q) * u])


def _stage(q, c, dt, p):
    """The conservative state after one Euler stage of length dt."""
    dx, dy = (p.xmax - p.xmin) / p.Nx, (p.ymax - p.ymin) / p.Ny
    P = _padded(q, p)
    C = P[:, 1:-1, 1:-1]
    sx = sy = torch.zeros_like(C)
    if p.reconstruction != fv.PCM:
        d = P[:, 1:-1, 1:] - P[:, 1:-1, :-1]
        sx = _minmod(d[:, :, :-1], d[:, :, 1:])
        d = P[:, 1:, 1:-1] - P[:, :-1, 1:-1]
        sy = _minmod(d[:, :-1], d[:, 1:])
    if p.reconstruction == fv.MUSCL_HANCOCK:
        (r, u, v, w), ax, ay = C, 0.5 * dt / dx, 0.5 * dt / dy
        C = C - torch.stack([
            ax * (u * sx[0] + r * sx[1]) + ay * (v * sy[0] + r * sy[2]),
            ax * (u * sx[1] + sx[3] / r) + ay * (v * sy[1]),
            ax * (u * sx[2]) + ay * (v * sy[2] + sy[3] / r),
            ax * (p.gamma0 * w * sx[1] + u * sx[3]) + ay * (p.gamma0 * w * sy[2] + v * sy[3])])
    swap = [0, 2, 1, 3]
    fx = _flux((C + 0.5 * sx)[:, 1:-1, :-1], (C - 0.5 * sx)[:, 1:-1, 1:], p, p.gx * dx)
    fy = _flux((C + 0.5 * sy)[swap, :-1, 1:-1], (C - 0.5 * sy)[swap, 1:, 1:-1], p, p.gy * dy)[swap]
    c = c + dt / dx * (fx[:, :, :-1] - fx[:, :, 1:]) + dt / dy * (fy[:, :-1] - fy[:, 1:])
    if p.gravity_mode == fv.GRAV_CONSTANT:
        for g, a, b in ((p.gx, fx[0][:, :-1], fx[0][:, 1:]), (p.gy, fy[0][:-1], fy[0][1:])):
            g = fv.as_float32(g)
            c[2] += dt * q[0] * g
            c[3] += dt * 0.5 * (a + b) * g
    if p.thermal_conductivity_active:
        T = P[3, 1:-1, 1:-1] / P[0, 1:-1, 1:-1]
        hx = p.kappa * (T[1:-1, 1:] - T[1:-1, :-1]) / dx
        hy = p.kappa * (T[1:, 1:-1] - T[:-1, 1:-1]) / dy
        c[3] += dt / dx * (hx[:, 1:] - hx[:, :-1]) + dt / dy * (hy[1:] - hy[:-1])
    if p.viscosity_active:
        u, v = P[1, 1:-1, 1:-1], P[2, 1:-1, 1:-1]
        mean = lambda a, axis: 0.5 * (a.narrow(axis, 1, a.shape[axis] - 1) + a.narrow(axis, 0, a.shape[axis] - 1))  # noqa: E731
        # x faces: gradients across the face, and along it from the four cells around
        ddx = lambda a: (a[1:-1, 1:] - a[1:-1, :-1]) / dx  # noqa: E731
        ady = lambda a: mean((a[2:] - a[:-2]) / (2.0 * dy), 1)  # noqa: E731
        txx, txy = 4.0 / 3.0 * ddx(u) - 2.0 / 3.0 * ady(v), ddx(v) + ady(u)
        ex = txx * mean(u, 1)[1:-1] + txy * mean(v, 1)[1:-1]
        ddy = lambda a: (a[1:, 1:-1] - a[:-1, 1:-1]) / dy  # noqa: E731
        adx = lambda a: mean((a[:, 2:] - a[:, :-2]) / (2.0 * dx), 0)  # noqa: E731
        tyy, tyx = 4.0 / 3.0 * ddy(v) - 2.0 / 3.0 * adx(u), ddy(u) + adx(v)
        ey = tyx * mean(u, 0)[:, 1:-1] + tyy * mean(v, 0)[:, 1:-1]
        # the step adds the face terms' differences times dt, without the spacing
        for k, a, b in ((1, txx, tyx), (2, txy, tyy), (3, ex, ey)):
            c[k] += dt * p.mu * ((a[:, 1:] - a[:, :-1]) + (b[1:] - b[:-1]))
    return c


def _dt(q, p):
    dx, dy = (p.xmax - p.xmin) / p.Nx, (p.ymax - p.ymin) / p.Ny
    a = torch.sqrt(p.gamma0 * q[3] / q[0])
    hyp = ((a + q[1].abs()) / dx + (a + q[2].abs()) / dy).max().item()
    least = min(dx, dy) ** 2
    tc = 2.0 * p.kappa / least if p.thermal_conductivity_active else p.epsilon
    visc = 2.0 * p.mu / least if p.viscosity_active else p.epsilon
    return p.CFL / max(hyp, tc, visc), hyp, tc, visc


def _march(q, p, steps):
    """Primitives (Ny, Nx, 4) after a number of steps from q (4, Ny, Nx), and the next dt."""
    gm1 = p.gamma0 - 1.0
    c = _cons(q, gm1)
    for _ in range(steps):
        dt = _dt(q, p)[0]
        n = _stage(q, c, dt, p)
        if p.time_stepping == fv.TS_RK2:
            n = 0.5 * (c + _stage(_prim(n, gm1), n, dt, p))
        c, q = n, _prim(n, gm1)
    return q.permute(1, 2, 0).contiguous(), _dt(q, p)[0]


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "served":
        return [_march(initial_values(p, v, device), p, steps)[0] for v, p, steps in _requests(case, seed)]
    p, q = _one(case, seed, device)
    q = q.permute(2, 0, 1).contiguous()
    if case["kind"] == "dt":
        return torch.tensor(_dt(q, p), dtype=torch.float64)
    prim, dt = _march(q, p, case["steps"])
    return dict(prim=prim.cpu().numpy() if case["kind"] == "host" else prim, dt=dt)
