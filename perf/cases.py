"""Performance cases: the work a user of this package has it do.

Four kinds of case, each through the entry point a program calls:

* ``grid``    -- one grid: state in from device tensors, ``steps`` RK3 steps, state out to device
                 tensors, time and next dt read back (``gpu.Solver``, what ``run.py`` does per snapshot);
* ``batch``   -- an ensemble of uneven grids, stepped as one batch with a replayed graph of all its steps;
* ``host``    -- one step on pinned host arrays (``Solver.step_host``: a host code's time loop);
* ``adjoint`` -- a differentiable run: forward, loss (magnetic energy), backward (``adjoint.run``).

Initial states are made here from the seed with plain torch: the benchmark problems (Orszag-Tang
vortex, rotor, Kelvin-Helmholtz shear, field loop, random smooth fields) with their parameters
jittered.  ``exact`` restates the scheme in plain 64-bit torch, whole array by whole array, in the
reference's order of operations: a limited state that rounds across its bound is reset to the cell's
value (MOOD), so a restatement that rounds otherwise resets other faces.
"""
from __future__ import annotations

import math

import torch

from chimera_b200 import adjoint, gpu
from chimera_b200.config import (BC_OUTFLOW, BC_PERIODIC, FP32_BULK, FP32_MIXED, FP64, HLLD, HLLE, MC, RUSANOV,
                                 VAN_LEER, SolverConfig)

_F64 = torch.float64
SOLVERS = {"rusanov": RUSANOV, "hlle": HLLE, "hlld": HLLD}
LIMITERS = {"mc": MC, "vanleer": VAN_LEER}
PRECISIONS = {"fp64": FP64, "fp32": FP32_BULK, "mixed": FP32_MIXED}
# periodic in (x, y); a side that is not periodic is outflow
SIDES = {"periodic": (True, True), "outflow": (False, False), "channel": (True, False)}


def _case(name, kind, flow, nx, ny, solver, limiter="mc", mood=True, sides="periodic", precision="fp64", steps=1,
          **more):
    return dict(name=name, kind=kind, flow=flow, nx=nx, ny=ny, solver=solver, limiter=limiter, mood=mood, sides=sides,
                precision=precision, steps=steps, **more)


def listed():
    return [
        # the smallest validation grid (Orszag-Tang 64^2, the reference's default switches): launches and latency
        _case("vortex64_fp64", "grid", "vortex", 64, 64, "rusanov", steps=10),
        # the reference's everyday size, Orszag-Tang 256^2
        _case("vortex256_fp64", "grid", "vortex", 256, 256, "rusanov", steps=20),
        # the headline workload: rotor 1024^2, outflow, HLLE
        _case("rotor1024_fp64", "grid", "rotor", 1024, 1024, "hlle", sides="outflow", steps=10),
        # Kelvin-Helmholtz with the costliest solver in FP64
        _case("shear2048_fp64", "grid", "shear", 2048, 2048, "hlld", steps=4),
        # odd sizes, dx != dy, Van Leer: a grid no tile shape and no tensor map fits
        _case("loop501x333_fp64", "grid", "loop", 501, 333, "hlle", limiter="vanleer", steps=10),
        # FP32 arithmetic on FP64 storage at the headline size
        _case("rotor1024_mixed", "grid", "rotor", 1024, 1024, "hlle", sides="outflow", precision="mixed", steps=10),
        # the largest grid: Kelvin-Helmholtz 4096^2, FP32-bulk
        _case("shear4096_fp32", "grid", "shear", 4096, 4096, "hlld", precision="fp32", steps=4),
        # an eighth of the random-field ensemble (128^2, 256^2, 512^2 members), FP32-bulk, and half that in FP64
        _case("ensemble_fp32", "batch", "random", 128, 128, "rusanov", precision="fp32", steps=20,
              members=32, doubled=24, quadrupled=8),
        _case("ensemble_fp64", "batch", "random", 128, 128, "rusanov", steps=10, members=16, doubled=12, quadrupled=4),
        # a host code's time loop: arrays in, one step, arrays out
        _case("host1024_fp64", "host", "rotor", 1024, 1024, "hlle", sides="outflow"),
        # gradients of a small run (sensitivity studies, the test size) and of the 512^2 field-loop workload
        _case("adjoint64", "adjoint", "random", 64, 64, "hlle", limiter="vanleer", steps=8, every=4),
        _case("adjoint512", "adjoint", "loop", 512, 512, "hlle", limiter="vanleer", steps=4, every=2),
    ]


_MAX_ZONES = {"grid": 2 ** 24, "batch": 2 ** 26, "host": 2 ** 21, "adjoint": 2 ** 20}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grid", "grid", "grid", "batch", "host", "adjoint", "adjoint"])
    top = {"grid": 3000, "batch": 256, "host": 1200, "adjoint": 600}[kind]
    nx = _log_int(rng, 24, top)
    ny = max(16, min(top, int(nx * rng.choice([1.0, 1.0, rng.uniform(0.4, 1.6)]))))
    if rng.random() < 0.4:   # sizes that a grid generator likes
        nx, ny = max(32, nx // 32 * 32), max(32, ny // 32 * 32)
    # gradients on states without exactly uniform regions, where every limiter sits at a kink
    flow = "random" if kind == "batch" else rng.choice(["loop", "random"] if kind == "adjoint" else
                                                       ["vortex", "rotor", "shear", "loop", "random"])
    case = dict(kind=kind, flow=flow, nx=nx, ny=ny, solver=rng.choice(list(SOLVERS)), limiter=rng.choice(list(LIMITERS)),
                mood=rng.random() < 0.8, precision="fp64", steps=1,
                sides="periodic" if kind == "batch" else rng.choice(["periodic", "periodic", "outflow", "channel"]))
    zones = nx * ny
    if kind == "batch":
        case["members"] = rng.randint(1, 24)
        case["doubled"] = rng.randint(0, 8)
        case["quadrupled"] = rng.randint(0, 2)
        zones *= case["members"] + 4 * case["doubled"] + 16 * case["quadrupled"]
    if kind in ("grid", "batch"):
        case["precision"] = rng.choice(["fp64", "fp64", "fp32", "mixed"])
    if kind != "host":
        case["steps"] = max(1, min(rng.randint(2, 16), _MAX_ZONES[kind] // zones))
    if kind == "adjoint":
        case["every"] = rng.randint(1, case["steps"])
    return case


# ---- configurations and initial states ---------------------------------------------------------


def _config(nx, ny, case, gamma):
    lx, ly = {"shear": (1.0, 2.0), "loop": (2.0, 1.0)}.get(case["flow"], (1.0, 1.0))
    px, py = SIDES[case["sides"]]
    bc = ((BC_PERIODIC if px else BC_OUTFLOW,) * 2) + ((BC_PERIODIC if py else BC_OUTFLOW,) * 2)
    return SolverConfig(nx=nx, ny=ny, dx=lx / nx, dy=ly / ny, gamma=gamma, bc=bc, t_end=1.0e30,
                        riemann=SOLVERS[case["solver"]], limiter=LIMITERS[case["limiter"]], mood=bool(case["mood"]),
                        precision=PRECISIONS[case["precision"]])


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _prev(f, dim, periodic):
    """The value at index i - 1 along dim; at i = 0 the far end or the cell itself."""
    n = f.shape[dim]
    return torch.cat([f.narrow(dim, n - 1 if periodic else 0, 1), f.narrow(dim, 0, n - 1)], dim)


def _next(f, dim, periodic):
    n = f.shape[dim]
    return torch.cat([f.narrow(dim, 1, n - 1), f.narrow(dim, 0 if periodic else n - 1, 1)], dim)


def _cell_field(f, dim, periodic):
    """Cell-centred B from a face component; at an outflow low side the face value itself (the mean
    of the face and itself)."""
    return 0.5 * (f + _prev(f, dim, periodic))


def _back_diff(f, dim, periodic, inv_h):
    """Backward difference along dim; at an outflow low side a copy of the next one."""
    d = (f - _prev(f, dim, periodic)) * inv_h
    if not periodic:
        n = f.shape[dim]
        d = torch.cat([d.narrow(dim, 1, 1), d.narrow(dim, 1, n - 1)], dim)
    return d


def _waves(X, Y, gen, lx, ly, modes=6, kmax=3):
    """A smooth random field: a few periodic waves of long wavelength."""
    f = torch.zeros_like(X)
    for _ in range(modes):
        k = torch.randint(-kmax, kmax + 1, (2,), generator=gen).tolist()
        if k == [0, 0]:
            k = [1, -1]
        phase, amp = (torch.rand(2, generator=gen, dtype=_F64) * 2.0 * math.pi).tolist()
        f = f + math.cos(amp) * torch.sin(2.0 * math.pi * (k[0] * X / lx + k[1] * Y / ly) + phase)
    return f


def _initial(case, nx, ny, seed):
    """(cfg, conserved state) of one grid: Mass, Momx, Momy, Energy, b_x, b_y, float64 (ny, nx)."""
    gen = torch.Generator().manual_seed(int(seed))
    u = torch.rand(8, generator=gen, dtype=_F64).tolist()
    dev = _device()
    flow = case["flow"]
    gamma = {"vortex": 5.0 / 3.0, "loop": 5.0 / 3.0, "random": 1.4 + 0.26 * u[0]}.get(flow, 1.4)
    cfg = _config(nx, ny, case, gamma)
    dx, dy = cfg.dx, cfg.dy
    lx, ly = dx * nx, dy * ny
    px, py = SIDES[case["sides"]]
    X = ((torch.arange(nx, dtype=_F64, device=dev) + 0.5) * dx)[None, :].expand(ny, nx)
    Y = ((torch.arange(ny, dtype=_F64, device=dev) + 0.5) * dy)[:, None].expand(ny, nx)
    one = torch.ones((ny, nx), dtype=_F64, device=dev)
    if flow == "vortex":   # Orszag-Tang, shifted
        Xs, Ys = 2.0 * math.pi * (X + u[1]), 2.0 * math.pi * (Y + u[2])
        rho, p = one * (25.0 / (36.0 * math.pi)), one * (5.0 / (12.0 * math.pi))
        vx, vy = -torch.sin(Ys), torch.sin(Xs)
        b0 = 1.0 / math.sqrt(4.0 * math.pi)
        Az = b0 * (torch.cos(2.0 * Xs) / (4.0 * math.pi) + torch.cos(Ys) / (2.0 * math.pi))
    elif flow == "rotor":   # a dense spinning disc in a uniform field
        rx, ry = X - (0.45 + 0.1 * u[1]), Y - (0.45 + 0.1 * u[2])
        r = torch.sqrt(rx * rx + ry * ry)
        f = torch.clamp((0.115 - r) / 0.015, 0.0, 1.0)
        rho, p = 1.0 + 9.0 * f, one
        w = (1.5 + u[3]) * f / torch.clamp(r, min=0.1)
        vx, vy = -w * ry, w * rx
        Az = (5.0 / math.sqrt(4.0 * math.pi)) * Y
    elif flow == "shear":   # two tanh layers and seeded noise
        s = Y - 1.0
        s = torch.where(s > 0.5, 1.0 - s, torch.where(s < -0.5, -1.0 - s, s))
        rho, p = one, 2.5 * one
        vx = 0.5 * torch.tanh(s / 0.05)
        noise = torch.rand((ny, nx), generator=torch.Generator(device=dev).manual_seed(int(seed)), dtype=_F64, device=dev)
        vy = 0.01 * torch.sin(2.0 * math.pi * (X + u[1])) * torch.exp(-s * s / 0.01) + 1.0e-3 * (2.0 * noise - 1.0)
        Az = 0.1 * (Y - 0.5 * ly)
    elif flow == "loop":   # a weak field loop carried by a nearly uniform flow
        r = torch.sqrt((X - (0.9 + 0.2 * u[1])) ** 2 + (Y - (0.45 + 0.1 * u[2])) ** 2)
        rho = 1.0 + 0.02 * _waves(X, Y, gen, lx, ly)
        p = 1.0 + 0.02 * _waves(X, Y, gen, lx, ly)
        vx, vy = 2.0 + 0.02 * _waves(X, Y, gen, lx, ly), 1.0 + 0.02 * _waves(X, Y, gen, lx, ly)
        Az = 1.0e-3 * torch.clamp(0.3 - r, min=0.0) + 1.0e-5 * _waves(X, Y, gen, lx, ly)
    else:   # random smooth velocity and field
        rho = 1.0 + 0.03 * _waves(X, Y, gen, lx, ly)
        p = 1.0 + 0.03 * _waves(X, Y, gen, lx, ly)
        vx, vy = _waves(X, Y, gen, lx, ly), _waves(X, Y, gen, lx, ly)
        vx, vy = ((0.5 + 0.8 * u[3]) * v / torch.sqrt(torch.mean(vx * vx + vy * vy)) for v in (vx, vy))
        Az = _waves(X, Y, gen, lx, ly) * (0.02 + 0.05 * u[4])
    b_x, b_y = _back_diff(Az, 0, py, 1.0 / dy), -_back_diff(Az, 1, px, 1.0 / dx)
    if flow in ("rotor", "shear"):   # A_z of a uniform field does not wrap
        b_x = torch.full_like(b_x, 5.0 / math.sqrt(4.0 * math.pi) if flow == "rotor" else 0.1)
    Bx, By = _cell_field(b_x, 1, px), _cell_field(b_y, 0, py)
    mass = rho * (dx * dy)
    energy = (p / (gamma - 1.0) + 0.5 * rho * (vx * vx + vy * vy) + 0.5 * (Bx * Bx + By * By)) * (dx * dy)
    return cfg, [t.contiguous() for t in (mass, mass * vx, mass * vy, energy, b_x, b_y)]


def _members(case, seed):
    """The grids of a case: one, or a batch's members."""
    sizes = [1] * case.get("members", 1) + [2] * case.get("doubled", 0) + [4] * case.get("quadrupled", 0)
    return [_initial(case, k * case["nx"], k * case["ny"], int(seed) + 1000003 * m) for m, k in enumerate(sizes)]


def _frozen_dt(cfg, U):
    """The time step of a differentiated run: fixed, below the CFL step of the initial state."""
    return 0.8 * _cfl(cfg, U)


# ---- the measured calls ------------------------------------------------------------------------


def prepare(case, seed):
    kind, steps = case["kind"], case["steps"]
    grids = _members(case, seed)
    cfg, U = grids[0]
    if kind == "adjoint":
        return dict(kind=kind, cfg=cfg, adj=adjoint.Adjoint(cfg), U=U, dts=[_frozen_dt(cfg, U)] * steps,
                    every=case["every"])
    solver = gpu.Solver([c for c, _ in grids])
    if kind == "host":
        out = [torch.empty(u.shape, dtype=_F64, pin_memory=True) for u in U]
        return dict(kind=kind, solver=solver, U=[u.cpu().pin_memory() for u in U], out=out)
    if kind == "batch":
        solver.set_graph_steps(steps)
    # results: the members' fields one after the other, one array per field
    final = [torch.empty(sum(c.cells for c, _ in grids), dtype=_F64, device=U[0].device) for _ in range(6)]
    parts = [f.split([c.cells for c, _ in grids]) for f in final]
    out = [[p[m].view(c.ny, c.nx) for p in parts] for m, (c, _) in enumerate(grids)]
    torch.cuda.synchronize()   # the solver has a stream of its own
    return dict(kind=kind, solver=solver, steps=steps, U=[st for _, st in grids], out=out, final=final)


def run(state):
    if state["kind"] == "adjoint":
        U0 = [u.detach().requires_grad_() for u in state["U"]]
        UN = adjoint.run(state["adj"], U0, state["dts"], K=state["every"])
        adjoint.magnetic_energy(state["cfg"], UN).backward()
        return {"final": [u.detach() for u in UN], "gradient": [u.grad for u in U0]}
    s = state["solver"]
    if state["kind"] == "host":
        s.set_time(0.0)
        return s.step_host(state["U"], out=state["out"])
    for m, st in enumerate(state["U"]):
        s.set_state(st, member=m)
        s.set_time(0.0, member=m)
    s.step(state["steps"])
    times = []
    for m, out in enumerate(state["out"]):
        s.get_state(member=m, out=out)
        d = s.diag(member=m)
        times.append((d["t"], d["dt"]))
    return {"final": state["final"], "time": torch.tensor(times, dtype=_F64)}


def work(case):
    """The state read and written once per step (its dt depends on the whole step before), the
    gradient's states and adjoints likewise; operations of the scheme's expressions per cell and RK
    stage (two faces of six limited fields, one Riemann solve each, the update), counted by hand."""
    k = [1] * case.get("members", 1) + [2] * case.get("doubled", 0) + [4] * case.get("quadrupled", 0)
    zones = sum(f * f for f in k) * case["nx"] * case["ny"] * case["steps"]
    word = 4 if case["precision"] == "fp32" else 8
    flops = {"rusanov": 620, "hlle": 680, "hlld": 900}[case["solver"]] * 3
    if case["kind"] == "adjoint":   # forward, recomputation and about two forwards' worth in reverse
        return {"bytes": zones * 8 * 6 * 6, "flops": zones * flops * 4}
    return {"bytes": zones * word * 12, "flops": zones * flops}


# ---- the scheme in plain 64-bit torch -----------------------------------------------------------


def _over(a, s):
    """a / s, rounded once (torch on CUDA multiplies by the reciprocal of a Python scalar)."""
    return a / torch.full((), s, dtype=_F64, device=a.device)


def _per(cfg):
    return cfg.bc[0] == BC_PERIODIC, cfg.bc[2] == BC_PERIODIC


def _primitives(cfg, U):
    px, py = _per(cfg)
    M, Mx, My, E, bx, by = U
    vol = cfg.dx * cfg.dy
    Bx, By = _cell_field(bx, 1, px), _cell_field(by, 0, py)
    rho = torch.clamp(_over(M, vol), min=1e-12)
    u, v = Mx / (rho * vol), My / (rho * vol)
    hb = 0.5 * (Bx * Bx + By * By)
    ke = 0.5 * rho * (u * u + v * v)
    P = torch.clamp((_over(E, vol) - ke - hb) * (cfg.gamma - 1.0) + hb, min=1e-12)
    return [rho, u, v, torch.maximum(P, hb + 1e-10 * (ke + hb)), Bx, By]


def _cfl(cfg, U):
    rho, u, v, P, Bx, By = _primitives(cfg, U)
    B2 = Bx * Bx + By * By
    inv = 1.0 / rho
    cf = torch.sqrt(cfg.gamma * (P - 0.5 * B2) * inv + B2 * inv)
    cf = torch.where(rho < 1e-3, torch.clamp(cf, max=50.0), cf)
    return cfg.courant * (min(cfg.dx, cfg.dy) / float((cf + torch.sqrt(u * u + v * v)).max()))


def _slope(dl, dr, limiter):
    den = dl + dr
    zero = (dl * dr <= 0.0) | (den.abs() < 1e-12)
    if limiter == VAN_LEER:
        s = 2.0 * (dl * dr) / torch.where(zero, torch.ones_like(den), den)
    else:
        s = torch.sign(dl) * torch.minimum(2.0 * torch.minimum(dl.abs(), dr.abs()), 0.5 * den.abs())
    return torch.where(zero, torch.zeros_like(s), s)


def _face_states(cfg, prim, dim):
    """Left and right states at the high face of every cell along dim."""
    px, py = _per(cfg)
    per, h = (px, cfg.dx) if dim == 1 else (py, cfg.dy)
    L, R = [], []
    for q, f in enumerate(prim):
        s = _slope((f - _prev(f, dim, per)) * (1.0 / h), (_next(f, dim, per) - f) * (1.0 / h), cfg.limiter)
        l, r = f + (0.5 * h) * s, _next(f - (0.5 * h) * s, dim, per)
        positive = q in (0, 3)
        if cfg.mood:   # both states held to the low cell's neighbourhood, or reset to its value
            near = [f, _next(f, 1, px), _prev(f, 1, px), _next(f, 0, py), _prev(f, 0, py)]
            lo, hi = near[0], near[0]
            for g in near[1:]:
                lo, hi = torch.minimum(lo, g), torch.maximum(hi, g)
            if positive:
                lo = torch.clamp(lo, min=1e-9)
            l, r = (torch.where((w < lo) | (w > hi), f, w) for w in (l, r))
        if positive:
            l, r = torch.clamp(l, min=1e-8), torch.clamp(r, min=1e-8)
        L.append(l)
        R.append(r)
    for S in (L, R):   # thermal pressure below the floor: the low cell's state
        bad = S[3] - 0.5 * (S[4] * S[4] + S[5] * S[5]) < 1e-12
        S[:] = [torch.where(bad, f, w) for f, w in zip(prim, S)]
    if dim == 0:
        L, R = ([S[0], S[2], S[1], S[3], S[5], S[4]] for S in (L, R))
    return L, R


def _physical(g, S, square_first=False):
    """Conserved variables, flux, thermal pressure and magnetic pressure of a face state
    (square_first: rho (u u) as the HLLD solver writes it)."""
    rho, u, v, P, Bn, Bt = S
    hb = 0.5 * (Bn * Bn + Bt * Bt)
    p = torch.clamp(P - hb, min=1e-12)
    e = _over(p, g - 1.0) + 0.5 * rho * (u * u + v * v) + hb
    ram = rho * (u * u) if square_first else rho * u * u
    F = [rho * u, ram + P - Bn * Bn, rho * u * v - Bn * Bt, (e + P) * u - Bn * (u * Bn + v * Bt),
         Bt * u - Bn * v]
    return [rho, rho * u, rho * v, e, Bt], F, p, hb


def _rusanov(g, L, R):
    UL, _, pL, hL = _physical(g, L)
    UR, _, pR, hR = _physical(g, R)
    rho, mx, my, e, Bt = (0.5 * (a + b) for a, b in zip(UL, UR))
    Bn = 0.5 * (L[4] + R[4])
    hb = 0.5 * (Bn * Bn + Bt * Bt)
    w = 1.0 / rho
    P = (g - 1.0) * (e - 0.5 * (mx * mx + my * my) * w - hb) + hb
    F = [mx, mx * mx * w + P - Bn * Bn, mx * my * w - Bn * Bt,
         (e + P) * mx * w - Bn * (Bn * mx + Bt * my) * w, (Bt * mx - Bn * my) * w]
    c = torch.maximum(torch.sqrt((g * pL + 2.0 * hL) / L[0]) + L[1].abs(),
                      torch.sqrt((g * pR + 2.0 * hR) / R[0]) + R[1].abs())
    return [f - (0.5 * c) * (b - a) for f, a, b in zip(F, UL, UR)]


def _hll(SL, SR, UL, UR, FL, FR):
    w = 1.0 / torch.clamp(SR - SL, min=1e-12)
    return [(SR * a - SL * b + SL * SR * (y - x)) * w for a, b, x, y in zip(FL, FR, UL, UR)]


def _hlle(g, L, R):
    UL, FL, pL, hL = _physical(g, L)
    UR, FR, pR, hR = _physical(g, R)
    cL = torch.clamp(torch.sqrt((g * pL + 2.0 * hL) / L[0]), max=100.0)
    cR = torch.clamp(torch.sqrt((g * pR + 2.0 * hR) / R[0]), max=100.0)
    SL, SR = torch.minimum(L[1] - cL, R[1] - cR), torch.maximum(L[1] + cL, R[1] + cR)
    F = _hll(SL, SR, UL, UR, FL, FR)
    return [torch.where(SR <= 0.0, b, torch.where(SL >= 0.0, a, f)) for f, a, b in zip(F, FL, FR)]


def _fast(g, S, p):
    c, a, b = (S[4] * S[4]) / S[0], g * p / S[0], (S[4] * S[4] + S[5] * S[5]) / S[0]
    t = a + b
    disc = torch.clamp(t * t - 4.0 * a * c, min=1e-300)
    return torch.clamp(torch.sqrt(0.5 * (t + torch.sqrt(disc))), max=50.0)


def _hlld(g, L, R):
    UL, FL, pL, _ = _physical(g, L, True)
    UR, FR, pR, _ = _physical(g, R, True)
    cL, cR = _fast(g, L, pL), _fast(g, R, pR)
    SL, SR = torch.minimum(L[1] - cL, R[1] - cR), torch.maximum(L[1] + cL, R[1] + cR)
    F_hll = _hll(SL, SR, UL, UR, FL, FR)
    wL, wR = L[0] * (SL - L[1]), R[0] * (SR - R[1])
    den = wR - wL
    den = torch.where(den.abs() < 1e-15, torch.copysign(torch.full_like(den, 1e-15), den), den)
    SM = (UR[1] * (SR - R[1]) - UL[1] * (SL - L[1]) - (R[3] - L[3])) / den
    narrow = (SM <= SL + 1e-6 * (SR - SL)) | (SM >= SR - 1e-6 * (SR - SL))
    one = torch.ones_like(SM)
    PT = torch.clamp(L[3] + wL * (SM - L[1]), min=1e-12)

    def star(S, U, w, speed):
        rho, u, v, P, Bn, Bt = S
        gap = torch.where(speed == SM, one, speed - SM)
        d = w * gap - Bn * Bn
        ok = d.abs() > 1e-3 * torch.clamp(torch.maximum((w * gap).abs(), Bn * Bn), min=1e-30)
        ds = torch.where(ok, d, one)
        vs = torch.where(ok, v - Bn * Bt * (SM - u) / ds, v)
        Bs = torch.where(ok, Bt * (rho * ((speed - u) * (speed - u)) - Bn * Bn) / ds, Bt)
        vB = SM * Bn + vs * Bs
        es = (U[3] * (speed - u) - P * u + PT * SM + Bn * (u * Bn + v * Bt - vB)) / gap
        rs = w / gap
        return [rs, rs * SM, rs * vs, es, Bs], vs, vB, torch.sqrt(torch.clamp(rs, min=1e-12))

    ULs, vLs, vBL, sL = star(L, UL, wL, SL)
    URs, vRs, vBR, sR = star(R, UR, wR, SR)
    Bn = 0.5 * (L[4] + R[4])
    on = Bn.abs() > 1e-10
    sg = torch.where(Bn < 0.0, -one, one)
    vss = torch.where(on, (sL * vLs + sR * vRs + sg * (URs[4] - ULs[4])) / (sL + sR), 0.5 * (vLs + vRs))
    Bss = torch.where(on, (sL * URs[4] + sR * ULs[4] + sg * sL * sR * (vRs - vLs)) / (sL + sR), 0.5 * (ULs[4] + URs[4]))
    vBss = SM * Bn + vss * Bss

    def side(U, F, Us, vs, vB, root, S, alfven, sign, inner):
        G = [f + S * (b - a) for f, a, b in zip(F, U, Us)]
        ess = torch.where(on, Us[3] + sign * (root * sg * (vB - vBss)), Us[3])
        more = [alfven * Us[0] * (vss - vs), alfven * (ess - Us[3]), alfven * (Bss - Us[4])]
        return G[:2] + [torch.where(inner, a + b, a) for a, b in zip(G[2:], more)]

    aL = torch.where(on, SM - Bn.abs() / sL, SM)
    aR = torch.where(on, SM + Bn.abs() / sR, SM)
    GL = side(UL, FL, ULs, vLs, vBL, sL, SL, aL, -1.0, aL < 0.0)
    GR = side(UR, FR, URs, vRs, vBR, sR, SR, aR, 1.0, aR > 0.0)
    G = [torch.where(SM >= 0.0, a, b) for a, b in zip(GL, GR)]
    top = torch.maximum(SL.abs(), SR.abs())
    wild = torch.zeros_like(narrow)
    for f, a, b, x, y in zip(G, FL, FR, UL, UR):
        wild = wild | ~torch.isfinite(f) | (f.abs() > 8.0 * (torch.maximum(a.abs(), b.abs()) + top * (x.abs() + y.abs())))
    G = [torch.where(wild | narrow, h, f) for f, h in zip(G, F_hll)]
    G = [torch.where(SL >= 0.0, a, torch.where(SR <= 0.0, b, f)) for f, a, b in zip(G, FL, FR)]
    capped = (cL >= 50.0) | (cR >= 50.0)
    return [torch.where(capped, torch.where(cL <= cR, a, b), f) for f, a, b in zip(G, FL, FR)]


_FLUX = {RUSANOV: _rusanov, HLLE: _hlle, HLLD: _hlld}


def _floors(cfg, U, Bx, By):
    M, Mx, My, E = U
    vol = cfg.dx * cfg.dy
    low = M < 1e-12 * vol
    E = torch.where(low, torch.maximum(E, (1e-12 / (cfg.gamma - 1.0) + 0.5 * (Bx * Bx + By * By)) * vol), E)
    Mx, My = (torch.where(low, torch.zeros_like(m), m) for m in (Mx, My))
    M = torch.where(low, torch.full_like(M, 1e-12 * vol), M)
    fast = Mx * Mx + My * My > (50.0 * M) ** 2
    mag = torch.sqrt(torch.where(fast, Mx * Mx + My * My, torch.ones_like(M)))
    Mx, My = (torch.where(fast, m * 50.0 * M / mag, m) for m in (Mx, My))
    return [M, Mx, My, E]


def _edge_inflow(cfg, prim, dim, a):
    """What enters the cells on an outflow low side in `a` = dt times the face: the physical flux of
    their own state (zero elsewhere): mass, x and y momentum, energy."""
    S = [f.narrow(dim, 0, 1) for f in prim]
    if dim == 0:
        S = [S[0], S[2], S[1], S[3], S[5], S[4]]
    rho, u, v, P, Bn, Bt = S
    hb = 0.5 * (Bn * Bn + Bt * Bt)
    e = _over(P - hb, cfg.gamma - 1.0) + 0.5 * rho * (u * u + v * v) + hb
    F = [a * rho * u, a * (rho * (u * u) + P - Bn * Bn), a * (rho * u * v - Bn * Bt),
         a * ((e + P) * u - Bn * (Bn * u + Bt * v))]
    if dim == 0:
        F = [F[0], F[2], F[1], F[3]]
    pad = list(prim[0].shape)
    pad[dim] -= 1
    zeros = torch.zeros(pad, dtype=_F64, device=prim[0].device)
    return [torch.cat([f, zeros], dim) for f in F]


def _stage(cfg, k, U, U0, dt):
    px, py = _per(cfg)
    prim = _primitives(cfg, U)
    Fx = _FLUX[cfg.riemann](cfg.gamma, *_face_states(cfg, prim, 1))
    Fy = _FLUX[cfg.riemann](cfg.gamma, *_face_states(cfg, prim, 0))
    Fy = [Fy[0], Fy[2], Fy[1], Fy[3], Fy[4]]
    new = []
    for q in range(4):
        f = U[q]
        for F, dim, per, a in ((Fx[q], 1, px, dt * cfg.dy), (Fy[q], 0, py, dt * cfg.dx)):
            inflow = _prev(F, dim, True)
            if not per:
                inflow = torch.cat([torch.zeros_like(F.narrow(dim, 0, 1)), F.narrow(dim, 0, F.shape[dim] - 1)], dim)
            f = f - a * F + a * inflow
        new.append(f)
    new = _floors(cfg, new, prim[4], prim[5])
    for dim, per, a in ((1, px, dt * cfg.dy), (0, py, dt * cfg.dx)):
        if not per:
            new = [f + c for f, c in zip(new, _edge_inflow(cfg, prim, dim, a))]
    Ez = 0.25 * (-Fx[4] - _next(Fx[4], 0, py) + Fy[4] + _next(Fy[4], 1, px))
    new.append(U[4] + dt * _back_diff(-Ez, 0, py, 1.0 / cfg.dy))
    new.append(U[5] - dt * _back_diff(-Ez, 1, px, 1.0 / cfg.dx))
    if k > 1:
        c = (0.75, 0.25) if k == 2 else (1.0 / 3.0, 2.0 / 3.0)
        new = [c[0] * a + c[1] * b for a, b in zip(U0, new)]
        new[:4] = _floors(cfg, new[:4], prim[4], prim[5])
    return new


def _step(cfg, U, dt):
    U1 = _stage(cfg, 1, U, U, dt)
    U2 = _stage(cfg, 2, U1, U, dt)
    return _stage(cfg, 3, U2, U, dt)


def _advance(cfg, U, steps):
    """`steps` CFL steps from t = 0, the step clipped to the output times: (state, t, next dt)."""
    t, count = 0.0, 1

    def next_dt():
        dt = _cfl(cfg, U)
        return max(count * cfg.t_out - t if t + dt > count * cfg.t_out else dt, float(torch.tensor(1e-12)))

    dt = next_dt()
    for _ in range(steps):
        U = _step(cfg, U, dt)
        t += dt
        count += t >= count * cfg.t_out
        dt = next_dt()
    return U, t, dt


def exact(case, seed):
    grids = _members(case, seed)
    cfg, U = grids[0]
    if case["kind"] == "adjoint":
        U0 = [u.detach().requires_grad_() for u in U]
        UN, dt = U0, _frozen_dt(cfg, U)
        for _ in range(case["steps"]):
            UN = _step(cfg, UN, dt)
        px, py = _per(cfg)
        Bx, By = _cell_field(UN[4], 1, px), _cell_field(UN[5], 0, py)
        (0.5 * torch.sum(Bx * Bx + By * By) * (cfg.dx * cfg.dy)).backward()
        return {"final": [u.detach() for u in UN], "gradient": [u.grad for u in U0]}
    if case["kind"] == "host":
        return [u.cpu() for u in _advance(cfg, U, 1)[0]]
    ends = [_advance(c, st, case["steps"]) for c, st in grids]
    return {"final": [torch.cat([U[q].flatten() for U, _, _ in ends]) for q in range(6)],
            "time": torch.tensor([(t, dt) for _, t, dt in ends], dtype=_F64)}
