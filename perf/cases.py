"""Workloads of the split 2D Euler solver, for timing it and checking its results.

Each case is work that a program using this package has it do through its
public entry points: whole solves through the reference's class, steps of a
state that stays on the GPU, many problems in a batch, and derivatives.
``exact`` restates the scheme in plain torch FP64, operation by operation in
the reference's order (src/basicFuns.cuh:13-274, src/wrappers.cuh:196-284).

Initial data: the package's workloads (seeded four-quadrant states, the
isentropic vortex, double Mach reflection, the shock-bubble) with smooth
seeded variations of every field, so that slopes are nonzero across the
domain, as they are once a flow has developed.
"""
import importlib
import math

import numpy as np
import torch

fvm = importlib.import_module("2d_fvm_cuda_b200")

OUTFLOW, DOUBLE_MACH, PERIODIC, REFLECTIVE_TB = 0, 4, 5, 6
PRECISION = {"fp64": fvm.FP64, "strict": fvm.FP64_STRICT, "fp32": fvm.FP32, "residual": fvm.FP32_RESIDUAL}
CFL, ALPHA, GAMMA = 0.45, 1.9, 1.4


def listed():
    return [
        # a parameter study on a small grid through the reference's class:
        # new four-quadrant states, setters kept, solve() to the end time;
        # launches, transfers and host work count here
        dict(name="class_solve_100", kind="class", nx=100, ny=100, t_end=0.05),
        # the 400 x 400 four-quadrant workload, state resident on the GPU,
        # a stretch of steps between two looks at the state
        dict(name="quadrant_400", kind="steps", flow="quadrant", nx=400, ny=400, steps=100, precision="fp64"),
        # double Mach reflection (n rows, about 4 n columns) at a ragged size
        dict(name="double_mach_131x517", kind="steps", flow="double_mach", nx=517, ny=131, steps=40, precision="fp64"),
        # smooth periodic flow at an odd size
        dict(name="vortex_1003", kind="steps", flow="vortex", nx=1003, ny=1003, steps=40, precision="fp64"),
        # the benchmark's size: a state far larger than the caches
        dict(name="quadrant_4096", kind="steps", flow="quadrant", nx=4096, ny=4096, steps=16, precision="fp64"),
        # the same in single precision with the compensated update
        dict(name="quadrant_4096_fp32", kind="steps", flow="quadrant", nx=4096, ny=4096, steps=16, precision="fp32"),
        # a shock running over a light bubble, walls above and below, single
        # precision with residual planes
        dict(name="bubble_2050x1025_residual", kind="steps", flow="bubble", nx=2050, ny=1025, steps=32,
             precision="residual"),
        # the reference's bits: a verification run
        dict(name="quadrant_400_strict", kind="steps", flow="quadrant", nx=400, ny=400, steps=60, precision="strict"),
        # an ensemble of uneven problems advanced together, each to its end time
        dict(name="batch_20_uneven", kind="batch", count=20, lo=64, hi=384, t_end=0.03, precision="fp64"),
        # gradient of a misfit of the final state, with checkpoints (inverse
        # problem at the size of the differentiation workload)
        dict(name="gradient_checkpoints_512", kind="gradient", nx=512, ny=512, steps=64, checkpoints=8),
        # the same with every step taped, at a ragged size
        dict(name="gradient_tape_243x310", kind="gradient", nx=243, ny=310, steps=40, checkpoints=0),
        # sensitivity of the final state in one direction
        dict(name="tangent_256x300", kind="tangent", nx=256, ny=300, steps=24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo_cells, hi_cells, lo=24, hi=4096):
    cells = math.exp(rng.uniform(math.log(lo_cells), math.log(hi_cells)))
    aspect = math.exp(rng.uniform(math.log(0.25), math.log(4.0)))
    nx = min(hi, max(lo, int(round(math.sqrt(cells * aspect)))))
    ny = min(hi, max(lo, int(round(math.sqrt(cells / aspect)))))
    return nx, ny


def draw(rng):
    kind = rng.choice(["class", "steps", "steps", "steps", "steps", "steps", "batch", "gradient", "gradient", "tangent"])
    if kind == "class":
        nx, ny = _sides(rng, 48 * 48, 256 * 256)
        return dict(kind=kind, nx=nx, ny=ny, t_end=round(rng.uniform(0.01, 0.06), 4))
    if kind == "steps":
        nx, ny = _sides(rng, 64 * 64, 4096 * 4096)
        flow = rng.choice(["quadrant", "quadrant", "vortex", "double_mach", "bubble"])
        # (a reflected shock amplifies rounding: fewer steps of it can be compared)
        most = 100 if flow in ("quadrant", "vortex") else 40
        steps = min(rng.randint(most // 2, most), max(4, int(16 * 4096 * 4096 / (nx * ny) * rng.uniform(0.3, 0.9))))
        precision = rng.choice(["fp64", "fp64", "fp64", "fp32", "fp32", "residual", "strict"])
        return dict(kind=kind, flow=flow, nx=nx, ny=ny, steps=steps, precision=precision)
    if kind == "batch":
        lo = _log_int(rng, 32, 128)
        return dict(kind=kind, count=rng.randint(6, 24), lo=lo, hi=rng.randint(lo + 32, 400),
                    t_end=round(rng.uniform(0.01, 0.03), 4), precision=rng.choice(["fp64", "fp32"]))
    if kind == "gradient":
        nx, ny = _sides(rng, 96 * 96, 512 * 512)
        steps = rng.randint(9, 64)
        return dict(kind=kind, nx=nx, ny=ny, steps=steps, checkpoints=rng.choice([0, max(2, round(math.sqrt(steps)))]))
    nx, ny = _sides(rng, 96 * 96, 400 * 400)
    return dict(kind="tangent", nx=nx, ny=ny, steps=rng.randint(4, 32))


# ---- inputs -------------------------------------------------------------------
def _waves(r, nx, ny, device):
    """A smooth field in [-1, 1]: three seeded Fourier modes."""
    x = torch.arange(nx, dtype=torch.float64, device=device) / nx
    y = torch.arange(ny, dtype=torch.float64, device=device) / ny
    w = torch.zeros(ny, nx, dtype=torch.float64, device=device)
    for _ in range(3):
        kx, ky = int(r.integers(1, 9)), int(r.integers(1, 9))
        px, py = float(r.uniform(0, 2 * math.pi)), float(r.uniform(0, 2 * math.pi))
        w += torch.sin(2 * math.pi * ky * y + py)[:, None] * torch.sin(2 * math.pi * kx * x + px)[None, :] / 3
    return w


def _vary(U, r, nx, ny, device, a=0.05):
    U[0] *= 1 + a * _waves(r, nx, ny, device)
    U[1] *= 1 + a * _waves(r, nx, ny, device)
    U[2] += a * _waves(r, nx, ny, device)
    U[3] += a * _waves(r, nx, ny, device)
    return U


def _quadrants(seed, nx, ny, device):
    U = torch.empty(4, ny, nx, dtype=torch.float64, device=device)
    q = fvm.scenarios.seeded_quadrant_states(seed)
    hx, hy = nx // 2, ny // 2
    for (rows, cols), s in zip([(slice(0, hy), slice(hx, nx)), (slice(0, hy), slice(0, hx)),
                                (slice(hy, ny), slice(0, hx)), (slice(hy, ny), slice(hx, nx))], q):
        for f in range(4):
            U[f, rows, cols] = s[f]
    return U


def _flow(flow, nx, ny, seed, device):
    """(planes (4, ny, nx), width, height, preset) of a flow."""
    r = np.random.default_rng([seed, 17])
    if flow == "quadrant":
        return _vary(_quadrants(seed, nx, ny, device), r, nx, ny, device), 1.0, ny / nx, OUTFLOW
    U = torch.empty(4, ny, nx, dtype=torch.float64, device=device)
    if flow == "vortex":
        h = 10.0 / (min(nx, ny) - 4)
        x = (torch.arange(nx, dtype=torch.float64, device=device) - 1.5) * h
        y = (torch.arange(ny, dtype=torch.float64, device=device) - 1.5) * h
        xc, yc, eps = float(r.uniform(4, 6)), float(r.uniform(4, 6)), float(r.uniform(3, 6))
        dx, dy = (x - xc)[None, :], (yc - y)[:, None]
        f = torch.exp(0.5 * (1.0 - dx * dx - dy * dy))
        T = 1.0 - (GAMMA - 1) * eps * eps / (8 * GAMMA * math.pi ** 2) * f * f
        U[0] = T ** (1 / (GAMMA - 1))
        U[1] = U[0] * T
        U[2] = 1.0 - eps / (2 * math.pi) * f * dy
        U[3] = 1.0 + eps / (2 * math.pi) * f * dx
        return _vary(U, r, nx, ny, device, 0.02), nx * h, ny * h, PERIODIC
    if flow == "double_mach":
        i = torch.arange(nx, device=device)[None, :]
        j = torch.arange(ny, device=device)[:, None]
        behind = i < ny // 6 + ((ny - j + 3) / math.sqrt(3.0)).to(torch.int64)
        for f in range(4):
            U[f] = fvm.scenarios.PRE_SHOCK_2MACH[f]
            U[f][behind] = fvm.scenarios.POST_SHOCK_2MACH[f]
        U[0] *= 1 + 0.05 * _waves(r, nx, ny, device)
        return U, float(nx) / ny, 1.0, DOUBLE_MACH
    assert flow == "bubble"
    rho2, p2, u2 = fvm.scenarios.mach2_post_shock(GAMMA)
    width, height = 2.0, 2.0 * ny / nx
    x = (torch.arange(nx, dtype=torch.float64, device=device) + 0.5) * (width / nx)
    y = (torch.arange(ny, dtype=torch.float64, device=device) + 0.5) * (height / ny)
    radius = 0.15 * min(1.0, height) * (1 + 0.1 * float(r.uniform(-1, 1)))
    inside = ((x - 0.4)[None, :] ** 2 + (y - height / 2)[:, None] ** 2) < radius * radius
    U[0], U[1], U[2], U[3] = 1.0, 1.0, 0.0, 0.0
    U[0][inside] = 0.1
    for f, v in ((0, rho2), (1, p2), (2, u2)):
        U[f][:, x < 0.1] = v
    U[0] *= 1 + 0.02 * _waves(r, nx, ny, device)
    U[2] += 0.1 * _waves(r, nx, ny, device)
    U[3] += 0.1 * _waves(r, nx, ny, device)
    return U, width, height, REFLECTIVE_TB


def _smooth(nx, ny, seed, device):
    """A smooth periodic flow whose fields vary everywhere, and its spacing's dt."""
    r = np.random.default_rng([seed, 29])
    U = torch.tensor([1.0, 1.0, 0.4, -0.3], dtype=torch.float64, device=device)[:, None, None].repeat(1, ny, nx)
    _vary(U, r, nx, ny, device, 0.2)
    h = min(1.0 / nx, 1.0 / ny)
    return U, 0.2 * h, r


def _batch_problems(case, seed):
    """[(planes on the CPU, nx, ny, t_end)] of a batch, sizes by the case alone."""
    sizes = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    out = []
    for k in range(case["count"]):
        nx, ny = (int(v) for v in sizes.integers(case["lo"], case["hi"] + 1, 2))
        U = _vary(_quadrants(seed * 1000 + k, nx, ny, "cpu"), np.random.default_rng([seed, k]), nx, ny, "cpu")
        out.append((U, nx, ny, case["t_end"]))
    return out


def _cells(planes):
    return np.ascontiguousarray(planes.cpu().numpy().transpose(1, 2, 0))


def _directions(r, nx, ny, device):
    return torch.stack([_waves(r, nx, ny, device) for _ in range(4)])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "class":
        s = fvm.RGRP_2D_CUDA()
        s.setSpatialLayout(1.0, case["ny"] / case["nx"])
        s.setTimeLayout(case["t_end"], CFL)
        return dict(case=case, solver=s, states=fvm.scenarios.seeded_quadrant_states(seed))
    if kind == "steps":
        U, width, height, preset = _flow(case["flow"], case["nx"], case["ny"], seed, "cuda")
        h = fvm.Handle(case["nx"], case["ny"])
        h.configure(width, height, 1e9, CFL, ALPHA, GAMMA, preset, PRECISION[case["precision"]])
        return dict(case=case, h=h, U=U, out=torch.empty_like(U))
    if kind == "batch":
        probs = _batch_problems(case, seed)
        b = fvm.Batch([(nx, ny) for _, nx, ny, _ in probs])
        b.set_precision(PRECISION[case["precision"]])
        for p, (_, nx, ny, t_end) in enumerate(probs):
            b.set_problem(p, 1.0, ny / nx, t_end, CFL, ALPHA, GAMMA, OUTFLOW)
        return dict(case=case, b=b, cells=[_cells(U) for U, _, _, _ in probs])
    U, dt, r = _smooth(case["nx"], case["ny"], seed, "cuda")
    h = fvm.Handle(case["nx"], case["ny"])
    h.configure(1.0, 1.0, 0.0, CFL, ALPHA, GAMMA, PERIODIC, fvm.FP64)
    h.set_fixed_dt(dt)
    d = _directions(r, case["nx"], case["ny"], "cuda")
    return dict(case=case, h=h, U=U, out=torch.empty_like(U), d=_cells(d))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "class":
        s = state["solver"]
        s.setRPInitialData(*state["states"], case["nx"], case["ny"])
        U = s.solve()
        return dict(rho=U[..., 0], p=U[..., 1], u=U[..., 2], v=U[..., 3])
    if kind == "steps":
        h, out = state["h"], state["out"]
        h.set_state_planes_ptr(state["U"].data_ptr())
        n = h.advance(case["steps"])
        h.get_state_planes_ptr(out.data_ptr())
        # single-precision builds: their fields go on as floats
        fields = out.float() if case["precision"] in ("fp32", "residual") else out
        return dict(rho=fields[0], p=fields[1], u=fields[2], v=fields[3], steps=n)
    if kind == "batch":
        b = state["b"]
        for p, U in enumerate(state["cells"]):
            b.set_state(p, U)
        b.solve()
        out = [b.get_state(p) for p in range(len(state["cells"]))]
        return [U.astype(np.float32) for U in out] if case["precision"] == "fp32" else out
    h, out = state["h"], state["out"]
    h.set_state_planes_ptr(state["U"].data_ptr())
    if kind == "tangent":
        tangent = h.jvp(case["steps"], state["d"])
        h.get_state_planes_ptr(out.data_ptr())
        return dict(state=out, tangent=tangent)
    h.forward(case["steps"], case["checkpoints"])
    gradient = h.vjp(state["d"])
    h.get_state_planes_ptr(out.data_ptr())
    return dict(state=out, gradient=gradient)


# ---- what a pass cannot do without --------------------------------------------
# per cell and step: the state read and written once; about 260 operations per
# cell in each of the four sweeps (three times that in a sweep's transpose,
# twice in a sweep that carries a tangent)
_FLOPS = 4 * 260


def work(case):
    kind = case["kind"]
    if kind == "batch":
        bytes_, flops = 0.0, 0.0
        word = 4 if case["precision"] == "fp32" else 8
        sizes = np.random.default_rng([case["count"], case["lo"], case["hi"]])
        for _ in range(case["count"]):
            nx, ny = (int(v) for v in sizes.integers(case["lo"], case["hi"] + 1, 2))
            steps = max(1.0, case["t_end"] * 3.5 * nx / CFL)
            bytes_ += nx * ny * (steps * 8 * word + 64)
            flops += nx * ny * steps * _FLOPS
        return dict(bytes=bytes_, flops=flops)
    cells = case["nx"] * case["ny"]
    if kind == "class":
        steps = max(1.0, case["t_end"] * 3.5 * case["nx"] / CFL)
        return dict(bytes=cells * (steps * 64.0 + 64), flops=cells * steps * _FLOPS)
    n = case["steps"]
    if kind == "steps":
        per = {"fp64": 64.0, "strict": 64.0, "fp32": 32.0, "residual": 48.0}[case["precision"]]
        return dict(bytes=cells * (n * per + 64), flops=float(cells) * n * _FLOPS)
    if kind == "tangent":
        return dict(bytes=cells * (n * 128.0 + 128), flops=float(cells) * n * 2 * _FLOPS)
    return dict(bytes=cells * (n * 192.0 + 128), flops=float(cells) * n * 4 * _FLOPS)


# ---- the scheme in plain torch FP64 ---------------------------------------------
def _slope(m, c, p, rh):
    central = (p - m) * 0.5 * rh
    back, fwd = (c - m) * rh * ALPHA, (p - c) * rh * ALPHA
    size = torch.minimum(central.abs(), torch.minimum(back.abs(), fwd.abs()))
    s = torch.where(central <= 0, -size, size)
    return torch.where((central * fwd > 0) & (back * fwd > 0), s, torch.zeros_like(s))


def _flux(L, R, sL, sR, k):
    """Relaxation GRP and midpoint flux: (mass, normal momentum, energy, tangential momentum)."""
    g = GAMMA
    rl, pl, ul, vl = L
    rr, pr, ur, vr = R
    rlx, plx, ulx, vlx = sL
    rrx, prx, urx, vrx = sR
    el, er = pl / rl / (g - 1), pr / rr / (g - 1)
    elx = plx / rl / (g - 1) - pl * rlx / rl / rl / (g - 1)
    erx = prx / rr / (g - 1) - pr * rrx / rr / rr / (g - 1)
    clx = 0.5 * torch.sqrt(g / pl / rl) * (pl * rlx + rl * plx)
    crx = 0.5 * torch.sqrt(g / pr / rr) * (pr * rrx + rr * prx)
    al, ar = torch.sqrt(g * pl / rl), torch.sqrt(g * pr / rr)
    kap = (g + 1) / 2
    pos = lambda v: torch.where(v > 0, v, torch.zeros_like(v))  # noqa: E731
    cl1 = rl * (al + kap * pos((pr - pl) / rr / ar + ul - ur))
    cr1 = rr * (ar + kap * pos((pl - pr) / cl1 + ul - ur))
    cr2 = rr * (ar + kap * pos((pl - pr) / rl / al + ul - ur))
    cl2 = rl * (al + kap * pos((pr - pl) / cr2 + ul - ur))
    up = pr >= pl
    cl, cr = torch.where(up, cl1, cl2), torch.where(up, cr1, cr2)
    um = (ul * cl + ur * cr + pl - pr) / (cl + cr)
    pm = ((ul - ur) * cl * cr + cl * pr + cr * pl) / (cl + cr)
    kl = -plx - cl * ulx + 0.5 * (0 - ul) * clx
    kr = -prx + cr * urx - 0.5 * (0 - ur) * crx
    dl = -2 * cl * cl / rl * ulx - 2 * cl / rl * plx + cl / rl * (0 - ul) * clx
    dr = 2 * cr * cr / rr * urx - 2 * cr / rr * prx + cr / rr * ur * crx
    Dp = (cr * dl - cl * dr) / 2 / (cl + cr)
    # right of the contact (um <= 0)
    a = cr / (ur - um + cr / rr)
    ea = er + (pm - pr) * (pm + pr) / 2 / cr / cr
    a_t = (-um * a * a * a / (rr * cr * cr) * (cr * cr / rr / rr * rrx - cr * urx + 1.5 * (um - ur) * crx)
           + a * a * a / (cr * cr * cr) * (um + cr / a) * Dp)
    ap_t = 1 / (cl + cr) * (cl * cr / rl * (1 + um * a / cr) * kl - cl * cr / rr * (1 - um * a / cl) * kr)
    au_t = 1 / (cl + cr) * (cl / rl * (1 + um * a / cr) * kl + cr / rr * (1 - um * a * cl / cr / cr) * kr)
    ae_t = (-um * a / rr / cr / cr / cr * (-pr * cr * prx + cr * cr * cr * erx + 2 * (er - ea) * cr * cr * crx)
            + pm / cr / cr * ap_t)
    # left of the contact (um > 0)
    b = cl / (um - ul + cl / rl)
    eb = el + (pm - pl) * (pm + pl) / 2 / cl / cl
    b_t = (-um * b * b * b / (rl * cl * cl) * (cl * cl / rl / rl * rlx + cl * ulx + 1.5 * (um - ul) * clx)
           - b * b * b / (cl * cl * cl) * (um - cl / b) * Dp)
    bp_t = 1 / (cl + cr) * (cl * cr / rl * (1 + um * b / cr) * kl - cl * cr / rr * (1 - um * b / cl) * kr)
    bu_t = 1 / (cl + cr) * (cl / rl * (1 + um * b * cr / cl / cl) * kl + cr / rr * (1 - um * b / cl) * kr)
    be_t = (-um * b / rl / cl / cl / cl * (-pl * cl * plx + cl * cl * cl * elx + 2 * (el - eb) * cl * cl * clx)
            + pm / cl / cl * bp_t)
    right = um <= 0
    star = (torch.where(right, a, b), pm, um, torch.where(right, vr, vl), torch.where(right, ea, eb),
            torch.where(right, a_t, b_t), torch.where(right, ap_t, bp_t), torch.where(right, au_t, bu_t),
            torch.where(right, -um * (a / rr * vrx), -um * (b / rl * vlx)), torch.where(right, ae_t, be_t))
    left = (rl, pl, ul, vl, el, -rl * ulx - ul * rlx, -ul * plx - cl * cl / rl * ulx, -ul * ulx - plx / rl, -ul * vlx,
            -ul * elx - pl / rl * ulx)
    rght = (rr, pr, ur, vr, er, -rr * urx - ur * rrx, -ur * prx - cr * cr / rr * urx, -ur * urx - prx / rr, -ur * vrx,
            -ur * erx - pr / rr * urx)
    to_right, to_left = ul - cl / rl >= 0, ur + cr / rr <= 0
    r, p, u, v, e, r_t, p_t, u_t, v_t, e_t = (torch.where(to_right, x, torch.where(to_left, y, z))
                                              for x, y, z in zip(left, rght, star))
    return (r * u + k / 2 * (r * u_t + u * r_t),
            r * u * u + p + k / 2 * (r_t * u * u + 2 * r * u * u_t + p_t),
            r * u * (e + u * u / 2 + v * v / 2) + p * u
            + k / 2 * (r_t * u * e + r * u_t * e + r * u * e_t + r_t * u * u * u / 2 + 1.5 * r * u * u * u_t
                       + r_t * u * v * v / 2 + r * u * v * v_t + r * u_t * v * v / 2 + p_t * u + p * u_t),
            r * u * v + k / 2 * (r * u_t * v + u * r_t * v + u * r * v_t))


def _sweep(W, h, dt):
    """Sweep along the last axis of W = (rho, p, un, ut), each (lines, n)."""
    g = GAMMA
    s = [_slope(w[:, :-2], w[:, 1:-1], w[:, 2:], 1.0 / h) for w in W]  # cells 1 .. n-2
    L = [w[:, 1:-2] + q[:, :-1] * h * 0.5 for w, q in zip(W, s)]
    R = [w[:, 2:-1] - q[:, 1:] * h * 0.5 for w, q in zip(W, s)]
    F = _flux(L, R, [q[:, :-1] for q in s], [q[:, 1:] for q in s], dt)
    lam = dt / h
    r, p, u, v = (w[:, 2:-2] for w in W)
    m = [r, r * u, p / (g - 1) + r * (u * u + v * v) / 2, r * v]
    m = [a - (f[:, 1:] - f[:, :-1]) * lam for a, f in zip(m, F)]
    new = [m[0], (g - 1) * (m[2] - m[1] * m[1] / m[0] / 2 - m[3] * m[3] / m[0] / 2), m[1] / m[0], m[3] / m[0]]
    return [torch.cat([w[:, :2], x, w[:, -2:]], 1) for w, x in zip(W, new)]


def _sweep_x(U, hx, dt):
    return _sweep(U, hx, dt)


def _sweep_y(U, hy, dt):  # along -j, with (un, ut) = (v, u)
    r, p, u, v = (w.flip(0).t() for w in U)
    r, p, v, u = _sweep([r, p, v, u], hy, dt)
    return [w.t().flip(0) for w in (r, p, u, v)]


def _ghost(U, preset, t):
    ny, nx = U[0].shape
    sign = [1.0, 1.0, 1.0, -1.0]
    out = []
    if preset == DOUBLE_MACH:
        post, pre = fvm.scenarios.POST_SHOCK_2MACH, fvm.scenarios.PRE_SHOCK_2MACH
        i = torch.arange(nx, device=U[0].device)
        top = i <= nx // 24 + int(ny / math.sqrt(3.0)) + int(ny * 20 * t / math.sqrt(3.0))
        foot = i <= nx // 24
        for f, w in enumerate(U):
            head = torch.full_like(w[:2], pre[f])
            head[:, top] = post[f]
            a = torch.where(foot, w[ny - 3], sign[f] * w[ny - 3])[None, :]
            b = torch.where(foot, w[ny - 3], sign[f] * w[ny - 4])[None, :]
            w = torch.cat([head, w[2:-2], a, b], 0)
            out.append(torch.cat([torch.full_like(w[:, :2], post[f]), w[:, 2:-2], torch.full_like(w[:, :2], pre[f])], 1))
        return out
    for f, w in enumerate(U):
        if preset == PERIODIC:
            w = torch.cat([w[ny - 4:ny - 2], w[2:-2], w[2:4]], 0)
            w = torch.cat([w[:, nx - 4:nx - 2], w[:, 2:-2], w[:, 2:4]], 1)
        else:
            if preset == REFLECTIVE_TB:
                w = torch.cat([sign[f] * w[3:4], sign[f] * w[2:3], w[2:-2], sign[f] * w[ny - 3:ny - 2],
                               sign[f] * w[ny - 4:ny - 3]], 0)
            else:
                w = torch.cat([w[2:3], w[2:3], w[2:-2], w[-3:-2], w[-3:-2]], 0)
            w = torch.cat([w[:, 2:3], w[:, 2:3], w[:, 2:-2], w[:, -3:-2], w[:, -3:-2]], 1)
        out.append(w)
    return out


def _step(U, hx, hy, dt, preset, t):
    A = _sweep_y(_sweep_x(U, hx, dt), hy, dt)
    B = _sweep_x(_sweep_y(U, hy, dt), hx, dt)
    return _ghost([(a + b) * 0.5 for a, b in zip(A, B)], preset, t + dt)


def _run_exact(U, width, height, preset, t_end, limit):
    """(fields, t, steps) after at most `limit` steps from t = 0."""
    U = list(U)
    ny, nx = U[0].shape
    hx, hy = width / nx, height / ny
    t, n = 0.0, 0
    while t < t_end and n < limit:
        smax = float((torch.sqrt(U[2] ** 2 + U[3] ** 2) + torch.sqrt(GAMMA * U[1] / U[0])).max())
        dt = min(CFL * min(hx, hy) / smax, t_end - t)
        U = _step(U, hx, hy, dt, preset, t)
        t, n = t + dt, n + 1
    return U, t, n


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "class":
            U = _quadrants(seed, case["nx"], case["ny"], "cuda")
            W, _, _ = _run_exact(U, 1.0, case["ny"] / case["nx"], OUTFLOW, case["t_end"], 1 << 30)
            return dict(zip(("rho", "p", "u", "v"), (w.cpu().numpy() for w in W)))
        if kind == "steps":
            U, width, height, preset = _flow(case["flow"], case["nx"], case["ny"], seed, "cuda")
            W, _, n = _run_exact(U, width, height, preset, 1e9, case["steps"])
            return dict(zip(("rho", "p", "u", "v"), W), steps=n)
        if kind == "batch":
            out = []
            for U, nx, ny, t_end in _batch_problems(case, seed):
                W, _, _ = _run_exact(U.cuda(), 1.0, ny / nx, OUTFLOW, t_end, 1 << 30)
                out.append(torch.stack(W, -1).cpu().numpy())
            return out
        U, dt, r = _smooth(case["nx"], case["ny"], seed, "cuda")
        d = _directions(r, case["nx"], case["ny"], "cuda")
        hx, hy = 1.0 / case["nx"], 1.0 / case["ny"]
        one = lambda *w: tuple(_step(list(w), hx, hy, dt, PERIODIC, 0.0))  # noqa: E731
        W = tuple(U)
        if kind == "tangent":
            D = tuple(d)
            for _ in range(case["steps"]):
                W, D = torch.func.jvp(one, W, D)
            return dict(state=torch.stack(W), tangent=torch.stack(D, -1).cpu().numpy())
        kept = []
        for _ in range(case["steps"]):
            kept.append(W)
            W = one(*W)
    G = tuple(d)
    for w in reversed(kept):
        w = tuple(x.clone().requires_grad_(True) for x in w)
        with torch.enable_grad():
            G = torch.autograd.grad(one(*w), w, G)
    return dict(state=torch.stack(W), gradient=torch.stack(G, -1).cpu().numpy())
