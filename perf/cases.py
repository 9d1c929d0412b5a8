"""Timing cases of the framework: the calls its users make, through the public entry points.

A case is a dict of plain values.  `kind` says which call it is:

  step      evolve() on a grid held on the GPU (FP64 forms "fp64" and "split", FP32 storage)
  ensemble  the replayed CUDA graph of an Ensemble (two time steps of every member)
  adjoint   rollout() forward, a misfit of the final state, and the gradient with
            respect to the initial state
  host      evolve_host(): one time step of a state that lives in host memory
  diag      compute_stats() and compute_solution_variables(), the diagnostics of a running simulation

The state is a flow in full motion (bubbles, wind and sound waves everywhere,
made from the seed), not the resting initial condition of the first step.  A
pass advances the state it is given, as a time loop does.

The literal FP64 form (f64_mode "native") is kept by the package as a check of
the others and is not timed here.
"""
import math

import numpy as np
import torch

from pyminiweather_gb300 import adjoint, ensemble, post
from pyminiweather_gb300.data import initialize_fields
from pyminiweather_gb300.ics import init
from pyminiweather_gb300.solve import evolve, evolve_host
from pyminiweather_gb300.solve import step as step_module

XLEN, ZLEN = 2e4, 1e4
STEP = dict(kind="step", ic="thermal", form="fp64", calls=1, nsteps=1)


def listed():
    return [
        # The reference's own example grid, one step: what each turn of an interactive time loop waits for.
        dict(STEP, name="thermal-100x50-fp64", nx=100, nz=50),
        # The command line's default grid and its default run of ten steps, one evolve() call a step as the driver does.
        dict(STEP, name="current-200x100-fp64-loop", ic="density-current", nx=200, nz=100, calls=10),
        # Odd sizes and the forcing term: a gravity-wave study, several steps a call.
        dict(STEP, name="gravity-401x199-fp64", ic="gravity", nx=401, nz=199, nsteps=8),
        # The benchmark's grid in the default form.
        dict(STEP, name="collision-8192x4096-fp64", ic="collision", nx=8192, nz=4096),
        # The same in the FP32 precision form.
        dict(STEP, name="collision-8192x4096-fp32", ic="collision", form="fp32", nx=8192, nz=4096),
        # FP32 on a grid whose rows are not 16-byte aligned, near the size of the reference's usage example.
        dict(STEP, name="thermal-2501x1251-fp32", form="fp32", nx=2501, nz=1251, nsteps=2),
        # The reference's usage example (2500 x 1250) in the double-FP32 form.
        dict(STEP, name="current-2500x1250-split", ic="density-current", form="split", nx=2500, nz=1250),
        # The benchmark's ensemble of 256 uneven members, FP32.
        dict(name="ensemble-256-fp32", kind="ensemble", form="fp32", members=256, lo=64, hi=1024, sizes=0),
        # A smaller FP64 ensemble of small members (a parameter sweep).
        dict(name="ensemble-48-fp64", kind="ensemble", form="fp64", members=48, lo=64, hi=512, sizes=1),
        # A gradient of the benchmark's adjoint configuration over 40 steps.
        dict(name="adjoint-512x256-fp64", kind="adjoint", form="fp64", nx=512, nz=256, nsteps=40, ckpt=20),
        # A host model's step: state in pinned host memory, copied in and out.
        dict(name="host-2048x1024-fp64", kind="host", form="fp64", nx=2048, nz=1024),
        # What a driver prints and writes at an output step.
        dict(name="diag-4096x2048-fp64", kind="diag", form="fp64", nx=4096, nz=2048),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("step", "step", "step", "step", "ensemble", "adjoint", "host", "diag"))
    if kind == "ensemble":
        return dict(kind=kind, form=rng.choice(("fp64", "fp32", "split")), members=log_int(8, 160), lo=rng.randint(24, 96),
                    hi=rng.randint(128, 768), sizes=rng.randint(2, 1 << 20))
    if kind == "adjoint":
        nx, n = log_int(48, 640), rng.randint(6, 40)
        return dict(kind=kind, form=rng.choice(("fp64", "split")), nx=nx, nz=max(8, nx * rng.randint(3, 8) // 10),
                    nsteps=n, ckpt=rng.randint(3, 20))
    if kind == "host":
        nx = log_int(128, 3000)
        return dict(kind=kind, form=rng.choice(("fp64", "split")), nx=nx, nz=max(16, nx * rng.randint(3, 8) // 10))
    if kind == "diag":
        nx = log_int(100, 5000)
        return dict(kind=kind, form=rng.choice(("fp64", "fp32")), nx=nx, nz=max(16, nx * rng.randint(3, 8) // 10))
    nx = log_int(40, 6000)
    return dict(STEP, ic=rng.choice(("thermal", "collision", "density-current", "gravity")),
                form=rng.choice(("fp64", "fp64", "fp32", "fp32", "split")), nx=nx, nz=max(12, nx * rng.randint(3, 8) // 10),
                calls=rng.choice((1, 1, 4)), nsteps=rng.choice((1, 1, 3)) if nx > 2000 else rng.randint(1, 8))


# ---- inputs -----------------------------------------------------------------------------------

GRAV, CP, CV, RD = 9.8, 1004.0, 717.0, 287.0
C0, GAMMA, P0, THETA0 = 27.5629410929725921310572974482, 1.40027894002789400278940027894, 1.0e5, 300.0
HV_BETA = 0.05


def device():
    return torch.device("cuda", torch.cuda.current_device())


def params_of(nx, nz, ic="thermal", form="fp64"):
    p = dict(nx=nx, nz=nz, xlen=XLEN, zlen=ZLEN, hs=2, s=4, ic_type=ic, cfl=1.5, max_speed=450.0)
    p["dx"], p["dz"] = XLEN / nx, ZLEN / nz
    p["dt"] = min(p["dx"], p["dz"]) * p["cfl"] / p["max_speed"]
    if form != "fp32":
        p["f64_mode"] = form
    return p


def dtype_of(case):
    return torch.float32 if case["form"] == "fp32" else torch.float64


def hydro(z, ic):
    """Density and potential temperature of the hydrostatic background at heights z."""
    if ic == "gravity":  # constant Brunt-Vaisala frequency
        n2 = 0.02 * 0.02
        t = THETA0 * torch.exp(n2 / GRAV * z)
        exner = 1.0 - GRAV * GRAV / (CP * n2) * (t - THETA0) / (t * THETA0)
    else:
        t = torch.full_like(z, THETA0)
        exner = 1.0 - GRAV * z / (CP * THETA0)
    return torch.pow(P0 * torch.pow(exner, CP / RD) / C0, 1.0 / GAMMA) / t, t


def flow(nx, nz, ic, rng, out_dtype):
    """(4, nz+4, nx+4): bubbles of the case, wind, density and sound waves in a few random modes."""
    dev, dx, dz = device(), XLEN / nx, ZLEN / nz
    x = ((torch.arange(nx + 4, dtype=torch.float64, device=dev) - 1.5) * dx)[None, :]
    z = ((torch.arange(nz + 4, dtype=torch.float64, device=dev) - 1.5) * dz)[:, None]
    r, _ = hydro(z, ic)
    amps = dict(thermal=[3.0], collision=[20.0, -20.0], gravity=[])
    amps["density-current"] = [-20.0]
    theta = torch.zeros(nz + 4, nx + 4, dtype=torch.float64, device=dev)
    for a in amps[ic]:
        x0, z0, rad = rng.uniform(0.3, 0.7) * XLEN, rng.uniform(0.25, 0.7) * ZLEN, rng.uniform(1500.0, 2500.0)
        d = torch.sqrt(((x - x0) / rad) ** 2 + ((z - z0) / rad) ** 2) * (math.pi / 2)
        theta += torch.where(d <= math.pi / 2, a * rng.uniform(0.8, 1.0) * torch.cos(d) ** 2, torch.zeros_like(d))

    def modes(amp, wall):
        f = torch.zeros(nz + 4, nx + 4, dtype=torch.float64, device=dev)
        for _ in range(3):
            kx, kz, ph = int(rng.integers(1, 5)), int(rng.integers(1, 4)), rng.uniform(0.0, 2 * math.pi)
            v = (torch.sin if wall else torch.cos)(kz * math.pi * z / ZLEN)
            f += amp * rng.uniform(0.3, 1.0) * torch.sin(2 * math.pi * kx * x / XLEN + ph) * v
        return f

    u = modes(3.0, False) + (15.0 if ic == "gravity" else 0.0)
    w = modes(1.0, True)
    rho = r * modes(1e-4, False)
    theta += modes(0.1, False)
    return torch.stack([rho, (r + rho) * u, (r + rho) * w, r * theta]).to(out_dtype)


def member_sizes(case):
    rng = np.random.default_rng(case["sizes"])
    n = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["members"]))
    return [(int(v), int(v) // 2) for v in np.rint(n)]


def prepare(case, seed):
    rng = np.random.default_rng([int(seed), 77])
    kind, dt = case["kind"], dtype_of(case)
    if kind == "ensemble":
        sizes = member_sizes(case)
        members = [(ensemble.member_params(nx, nz), None) for nx, nz in sizes]
        e = ensemble.Ensemble(members, dtype=dt, f64_mode="fp64" if case["form"] == "fp32" else case["form"])
        for k, (nx, nz) in enumerate(sizes):
            e.member_state(k).copy_(flow(nx, nz, "thermal", rng, dt))
        e.state_tmp.copy_(e.state)
        return dict(kind=kind, ens=e, replay=e.graph())
    nx, nz, ic = case["nx"], case["nz"], case.get("ic", "thermal")
    p = params_of(nx, nz, ic, case["form"])
    f = initialize_fields(p, dtype=dt)
    init(f, p)
    state = flow(nx, nz, ic, rng, dt)
    if kind == "adjoint":
        target = flow(nx, nz, ic, rng, dt)
        return dict(kind=kind, p=p, state=state, target=target, nz=nz,
                    ctx=adjoint.RolloutContext(params=p, fields=f, nsteps=case["nsteps"], ckpt_every=case["ckpt"]))
    f.state.copy_(state)
    f.state_tmp.copy_(state)
    s = dict(kind=kind, p=p, f=f, reverse=False, calls=case.get("calls", 1), nsteps=case.get("nsteps", 1))
    if kind == "host":
        s["h"] = state.cpu().pin_memory()
        s["h_out"] = torch.empty_like(s["h"]).pin_memory()
    return s


def run(s):
    kind = s["kind"]
    if kind == "ensemble":
        s["replay"]()
        return dict(state=s["ens"].state, state_tmp=s["ens"].state_tmp)
    if kind == "adjoint":
        x0 = s["state"].requires_grad_(True)
        end = adjoint.rollout(x0, s["ctx"])
        loss = adjoint.upper_half_rhot_misfit(end, s["target"], s["nz"])
        (g,) = torch.autograd.grad(loss, x0)
        return dict(state=end, loss=loss, grad=g)
    p, f = s["p"], s["f"]
    if kind == "diag":
        mass, energy = post.compute_stats(p, f)
        return dict(mass=mass, energy=energy, variables=post.compute_solution_variables(p, f))
    # each simulation keeps its own place in the alternation of the two directions
    step_module.reset_direction(s["reverse"])
    if kind == "host":
        evolve_host(p, f, s["h"], s["h_out"], dt=p["dt"])
        s["reverse"] = step_module.reverse_direction
        return dict(state=s["h_out"])
    for _ in range(s["calls"]):
        evolve(p, f, None, dt=p["dt"], nsteps=s["nsteps"])
    s["reverse"] = step_module.reverse_direction
    return dict(state=f.state, state_tmp=f.state_tmp)


# ---- what a pass cannot do without --------------------------------------------------------------

# Operations of one cell in one direction and RK stage: per variable the 4-point interpolation, the third
# difference and the update (5 + 2), the flux with its reciprocal and the pressure's power (about 30).
FLOPS_CELL_STAGE = 4 * 7 + 30


def work(case):
    kind, b = case["kind"], 4 if case["form"] == "fp32" else 8
    if kind == "ensemble":
        cells = sum(nx * nz for nx, nz in member_sizes(case))
        return dict(bytes=2 * 3 * 4 * b * cells, flops=2 * 6 * FLOPS_CELL_STAGE * cells)
    cells = case["nx"] * case["nz"]
    if kind == "adjoint":  # forward, and in reverse each step's stages again and their transposes
        n = case["nsteps"]
        return dict(bytes=n * 4 * b * cells * 4, flops=n * 6 * FLOPS_CELL_STAGE * cells * 4)
    if kind == "diag":
        return dict(bytes=(2 * 4 * b if b == 8 else 4 * (b + 8)) * cells, flops=60 * cells)
    n = case.get("calls", 1) * case.get("nsteps", 1)  # per step: the state read and written, state_tmp written
    return dict(bytes=n * 3 * 4 * b * cells, flops=n * 6 * FLOPS_CELL_STAGE * cells)


# ---- the same results from plain torch in 64 bits -----------------------------------------------


def backgrounds(nz, ic):
    dev, dz = device(), ZLEN / nz
    zc = (torch.arange(nz + 4, dtype=torch.float64, device=dev) - 1.5) * dz
    zi = torch.arange(nz + 1, dtype=torch.float64, device=dev) * ((nz + 1) * dz / (nz + 1))
    rc, tc = hydro(zc, ic)
    ri, ti = hydro(zi, ic)
    return rc, rc * tc, ri, ri * ti, C0 * torch.pow(ri * ti, GAMMA)


def source(nx, nz, bg):
    dev, dx, dz = device(), XLEN / nx, ZLEN / nz
    x = (dx / 2 + torch.arange(nx, dtype=torch.float64, device=dev) * dx)[None, :]
    z = (dz / 2 + torch.arange(nz, dtype=torch.float64, device=dev) * dz)[:, None]
    d = torch.sqrt(((x - XLEN / 8) / 500.0) ** 2 + ((z - 1000.0) / 500.0) ** 2) * (math.pi / 2)
    return torch.where(d <= math.pi / 2, 0.01 * torch.cos(d) ** 2, torch.zeros_like(d)) * bg[0][2:-2, None]


def fill_halo(q, bg, direction):
    """The halo a stage writes into the array it is forced by: periodic in x, solid walls in z."""
    if direction == "x":
        q[:, 2:-2, :2] = q[:, 2:-2, -4:-2]
        q[:, 2:-2, -2:] = q[:, 2:-2, 2:4]
        return
    for halo, row in (((0, 1), 2), ((-2, -1), -3)):
        for h in halo:
            q[0, h], q[3, h], q[2, h] = q[0, row], q[3, row], 0.0
            q[1, h] = q[1, row] / bg[0][row] * bg[0][h]


def tendency(q, bg, p, direction, src):
    """q: a halo-filled state; the tendency of its interior."""
    axis, d = (2, p["dx"]) if direction == "x" else (1, p["dz"])
    q = q[:, 2:-2, :] if direction == "x" else q[:, :, 2:-2]
    n = q.shape[axis] - 3
    s0, s1, s2, s3 = (q.narrow(axis, j, n) for j in range(4))
    v = (7.0 * (s1 + s2) - (s0 + s3)) / 12.0
    d3 = (s3 - s0) + 3.0 * (s1 - s2)
    hv = HV_BETA * d / (16.0 * p["dt"])
    rc, rtc, ri, rti, pri = bg
    if direction == "x":
        rho, rt, pb = v[0] + rc[2:-2, None], v[3] + rtc[2:-2, None], 0.0
        m = v[1]
    else:
        rho, rt, pb = v[0] + ri[:, None], v[3] + rti[:, None], pri[:, None]
        inside = torch.ones(n, 1, dtype=torch.float64, device=q.device)
        inside[0] = inside[-1] = 0.0
        m = v[2] * inside
        d3 = torch.cat([d3[:1] * inside, d3[1:]])
    un = m / rho
    pr = C0 * torch.pow(rt, GAMMA) - pb
    if direction == "x":
        f = torch.stack([m, un * v[1] + pr, un * v[2], un * rt]) + hv * d3
    else:
        f = torch.stack([m, un * v[1], un * m + pr, un * rt]) + hv * d3
    t = -(f.narrow(axis, 1, n - 1) - f.narrow(axis, 0, n - 1)) / d
    extra = torch.zeros_like(t[2])
    if direction == "z":
        extra = extra - GRAV * q[0, 2:-2]
    if src is not None:
        extra = extra + src
    return torch.cat([t[:2], (t[2] + extra)[None], t[3:]])


def plain_steps(s, tmp, bg, p, n, reverse=False, src=None, halo=True):
    """n time steps of the full arrays s and tmp, halos as a time loop leaves them (in place)."""
    inner = (slice(None), slice(2, -2), slice(2, -2))

    def stage(base, forcing, out, dt, direction):
        q = forcing if halo else forcing.clone()
        fill_halo(q, bg, direction)
        new = base[inner] + dt * tendency(q, bg, p, direction, src)
        out[inner] = new

    for _ in range(n):
        for d in ("x", "z") if reverse else ("z", "x"):
            stage(s, s, tmp, p["dt"] / 3, d)
            stage(s, tmp, tmp, p["dt"] / 2, d)
            stage(s, tmp, s, p["dt"], d)
        reverse = not reverse
    return reverse


def plain_gradient(x0, target, bg, p, n, nz):
    """The final state, the misfit and its gradient, by autograd through the interior steps."""

    def whole(s, direction):
        if direction == "x":
            q = torch.cat([s[:, :, -2:], s, s[:, :, :2]], 2)
            return torch.nn.functional.pad(q, (0, 0, 2, 2))
        z = torch.zeros_like(s[0, :1])
        rc = bg[0]

        def wall(row, h, src):
            return torch.stack([row[0], row[1] / rc[src] * rc[h], z[0], row[3]])[:, None]

        q = torch.cat([wall(s[:, 0], 0, 2), wall(s[:, 0], 1, 2), s, wall(s[:, -1], -2, -3), wall(s[:, -1], -1, -3)], 1)
        return torch.nn.functional.pad(q, (2, 2))

    def one(s, reverse):
        for d in ("x", "z") if reverse else ("z", "x"):
            s1 = s + p["dt"] / 3 * tendency(whole(s, d), bg, p, d, None)
            s2 = s + p["dt"] / 2 * tendency(whole(s1, d), bg, p, d, None)
            s = s + p["dt"] * tendency(whole(s2, d), bg, p, d, None)
        return s

    x = x0[:, 2:-2, 2:-2].clone().requires_grad_(True)
    s = x
    for k in range(n):
        s = torch.utils.checkpoint.checkpoint(one, s, bool(k % 2), use_reentrant=False)
    diff = (s[3] - target[3, 2:-2, 2:-2])[nz // 2:]
    loss = (diff * diff).sum()
    (g,) = torch.autograd.grad(loss, x)
    end, grad = x0.clone(), torch.zeros_like(x0)
    end[:, 2:-2, 2:-2] = s.detach()
    grad[:, 2:-2, 2:-2] = g
    return end, loss.detach(), grad


def exact(case, seed):
    rng = np.random.default_rng([int(seed), 77])
    kind, dt = case["kind"], dtype_of(case)
    if kind == "ensemble":
        states, tmps = [], []
        for nx, nz in member_sizes(case):
            s = flow(nx, nz, "thermal", rng, dt).double()
            t = s.clone()
            plain_steps(s, t, backgrounds(nz, "thermal"), params_of(nx, nz), 2)
            states.append(s.reshape(-1))
            tmps.append(t.reshape(-1))
        return dict(state=torch.cat(states), state_tmp=torch.cat(tmps))
    nx, nz, ic = case["nx"], case["nz"], case.get("ic", "thermal")
    p, bg = params_of(nx, nz, ic), backgrounds(nz, ic)
    s = flow(nx, nz, ic, rng, dt).double()
    if kind == "adjoint":
        target = flow(nx, nz, ic, rng, dt).double()
        end, loss, g = plain_gradient(s, target, bg, p, case["nsteps"], nz)
        return dict(state=end, loss=loss, grad=g)
    if kind == "diag":
        q = s[:, 2:-2, 2:-2]
        r, rt = bg[0][2:-2, None], bg[1][2:-2, None]
        rho = q[0] + r
        th = (q[3] + rt) / rho
        press = C0 * torch.pow(rho * th, GAMMA)
        energy = (q[1] ** 2 + q[2] ** 2) / rho + rho * CV * th / torch.pow(P0 / press, RD / CP)
        area = p["dx"] * p["dz"]
        return dict(mass=float(rho.sum() * area), energy=float(energy.sum() * area),
                    variables=torch.stack([q[0], q[1] / rho, q[2] / rho, th - rt / r]))
    t = s.clone()
    src = source(nx, nz, bg) if ic == "gravity" else None
    if kind == "host":
        plain_steps(s, t, bg, p, 1)
        return dict(state=s)
    plain_steps(s, t, bg, p, case["calls"] * case["nsteps"], src=src)
    return dict(state=s, state_tmp=t)
