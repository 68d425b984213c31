"""Performance cases of the finite-volume library: the calls its users make,
over the sizes they make them at.

Every case drives a public entry point of `bsn` on inputs made on the GPU from
a seed: a blast wave part of the way to the boundary (the Sedov and supernova
runs), a rotating polytrope in a floor atmosphere (the mesh-refined star), or
an exploding star between two black-hole sinks (the binary runs).  Entry
points that advance a state in place start each pass from the same state, as a
program restarting from a checkpoint does, so every pass does the same work.
`exact` restates the uniform-grid paths in plain torch in 64 bits.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "binary-supernova_b200"))

import bsn  # noqa: E402
from bsn import ics  # noqa: E402

NG = 3
DEV = "cuda"
F64 = torch.float64
#: floating-point operations of the scheme per cell and SSP-RK3 step
FLOPS_PER_CELL_STEP = 10023.0


# ---------------------------------------------------------------------------
# the cases

def listed():
    return [
        # the host-driven loop (dt, then a step) of a small validation run
        dict(name="step_f64_24", kind="step", precision="f64", nx=24, ny=24, nz=24, bc="outflow"),
        # the same loop with FP32 stencils on a ragged periodic box
        dict(name="step_f32_150x101x67", kind="step", precision="f32", nx=150, ny=101, nz=67, bc="periodic"),
        # the device time loop of a laptop-sized FP64 run
        dict(name="run_f64_64", kind="run", precision="f64", nx=64, ny=64, nz=64, bc="outflow", steps=4),
        # the production resolution of the uniform blast wave, in each of the three stencil forms
        dict(name="run_f64_256", kind="run", precision="f64", nx=256, ny=256, nz=256, bc="outflow", steps=1),
        dict(name="run_f32_256", kind="run", precision="f32", nx=256, ny=256, nz=256, bc="outflow", steps=2),
        dict(name="run_learned_256", kind="run", precision="learned", nx=256, ny=256, nz=256, bc="outflow", steps=2),
        # the right-hand side with its face fluxes, for a caller's own time integration
        dict(name="rhs_f64_90x61x47", kind="rhs", precision="f64", nx=90, ny=61, nz=47, bc="periodic"),
        # the isolated potential of a 128^3 density, in both transform precisions
        dict(name="poisson_f64_128", kind="poisson", precision="f64", nx=128, ny=128, nz=128),
        dict(name="poisson_f32_128", kind="poisson", precision="f32", nx=128, ny=128, nz=128),
        # the binary black-hole supernova on one uniform grid: orbit, sinks, self-gravity, diagnostics
        dict(name="coupled_f64_64", kind="coupled", precision="f64", n=64, self_gravity=True, steps=2),
        # the self-gravitating star on two mesh levels
        dict(name="fmr_f32_128", kind="fmr", precision="f32", n=128, self_gravity=True, steps=2),
        # the binary black-hole supernova on three nested mesh levels
        dict(name="nested_f32_128", kind="nested", precision="f32", n=128, self_gravity=True, steps=1),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "run", "run", "run", "rhs", "poisson", "coupled", "fmr", "nested"])
    prec = rng.choice(["f64", "f32", "learned"])
    if kind in ("step", "run"):
        n = [_logint(rng, 16, 224) for _ in range(3)]
        if kind == "run" and rng.random() < 0.5:    # the cubes of most runs
            n = [4 * _logint(rng, 6, 60)] * 3
        c = dict(kind=kind, precision=prec, nx=n[0], ny=n[1], nz=n[2], bc=rng.choice(["outflow", "periodic"]))
        if kind == "run":
            cells = n[0] * n[1] * n[2]
            c["steps"] = rng.randint(1, 8) if cells < 96 ** 3 else 1
        return c
    if kind == "rhs":
        n = [_logint(rng, 16, 128) for _ in range(3)]
        return dict(kind=kind, precision=rng.choice(["f64", "f32"]), nx=n[0], ny=n[1], nz=n[2],
                    bc=rng.choice(["outflow", "periodic"]))
    if kind == "poisson":
        n = [2 ** rng.randint(4, 8) for _ in range(3)]
        return dict(kind=kind, precision=rng.choice(["f64", "f32"]), nx=n[0], ny=n[1], nz=n[2])
    if kind == "coupled":
        sg = rng.random() < 0.7
        n = rng.choice([32, 64, 128]) if sg else _logint(rng, 24, 120)
        return dict(kind=kind, precision=prec, n=n, self_gravity=sg, steps=rng.randint(1, 2))
    # mesh levels: an even division of the base grid; self-gravity wants powers of two
    sg = rng.random() < 0.6
    n = rng.choice([32, 64, 128]) if sg else 4 * _logint(rng, 6, 28)
    return dict(kind=kind, precision=prec, n=n, self_gravity=sg, steps=1 if kind == "nested" else rng.randint(1, 2))


# ---------------------------------------------------------------------------
# inputs

def _centres(n, dx, x0, ghosts):
    g = NG if ghosts else 0
    return x0 + (torch.arange(-g, n + g, device=DEV, dtype=F64) + 0.5) * dx


def _ripple(xc, yc, zc, rng, scale):
    """A smooth field of order one: a few plane waves with seeded directions and phases."""
    out = 0.0
    for _ in range(3):
        k = rng.normal(size=3) * scale
        out = out + torch.sin(float(k[0]) * xc[None, None, :] + float(k[1]) * yc[None, :, None]
                              + float(k[2]) * zc[:, None, None] + float(rng.uniform(0, 6.28)))
    return out / 3.0


def _pack(rho, v, P, gamma):
    U = torch.empty(rho.shape + (5,), device=DEV, dtype=F64)
    U[..., 0] = rho
    ke = 0.0
    for q in range(3):
        U[..., q + 1] = rho * v[q]
        ke = ke + v[q] * v[q]
    U[..., 4] = P / (gamma - 1.0) + 0.5 * rho * ke
    return U.permute(3, 2, 1, 0)


def _blast(nx, ny, nz, gamma, seed):
    """A blast wave in uniform gas at rest: the self-similar interior's power
    laws behind a shock smeared over three cells, with a one per cent ripple."""
    rng = np.random.default_rng(seed)
    dx = 2.0 / max(nx, ny, nz)
    xc, yc, zc = (_centres(n, dx, -0.5 * n * dx, True) for n in (nx, ny, nz))
    c = rng.uniform(-0.05, 0.05, 3)
    X, Y, Z = (xc - float(c[0]))[None, None, :], (yc - float(c[1]))[None, :, None], (zc - float(c[2]))[:, None, None]
    r = torch.sqrt(X * X + Y * Y + Z * Z)
    # the shock: part of the way to the nearest boundary, decelerating as R^(-3/2)
    R = float(rng.uniform(0.3, 0.5)) * min(nx, ny, nz) / max(nx, ny, nz) + 2 * dx
    D = 0.6 * R ** -1.5
    s = ((R - r) / (3 * dx)).clamp(0.0, 1.0)
    s = s * s * (3 - 2 * s)
    x = (r / R).clamp(max=1.0)
    rip = 1.0 + 0.01 * _ripple(xc, yc, zc, rng, 12.0)
    rho = 1.0 + s * ((gamma + 1) / (gamma - 1) * x ** 4.5 * rip + 1e-3 - 1.0)
    P = 1e-5 + s * (2 / (gamma + 1) * D * D * (0.31 + 0.69 * x ** 8))
    vr = s * (2 / (gamma + 1) * D) * x * rip / r.clamp(min=1e-12)
    return _pack(rho, (vr * X, vr * Y, vr * Z), P, gamma), dx


_STAR = {}


def _polytrope(r, index, mass, radius, gamma, rho_floor, P_floor):
    """Density and pressure of a polytrope in a floor atmosphere."""
    if index not in _STAR:
        _STAR[index] = ics.lane_emden(index)
    xi, th, dth = _STAR[index]
    xi1, om = float(xi[-1]), -float(xi[-1]) ** 2 * float(dth[-1])
    rs = radius / xi1
    rho_c = mass / (4 * math.pi * rs ** 3 * om)
    K = 4 * math.pi * rs ** 2 * rho_c ** (1 - 1 / index) / (index + 1)
    t = torch.as_tensor(th, device=DEV, dtype=F64)
    f = (r / rs / float(xi[1] - xi[0]) - 1.0).clamp(0.0, len(xi) - 2 + 0.999)
    i = f.floor().long()
    theta = torch.lerp(t[i], t[i + 1], f - i)
    theta = torch.where(r < radius, theta.clamp(min=0.0), torch.zeros_like(theta))
    rho = rho_c * theta ** index
    inside = rho > rho_floor
    rho = torch.where(inside, rho, torch.full_like(rho, rho_floor))
    P = torch.where(inside, K * rho ** (1 + 1 / index), torch.full_like(rho, P_floor)).clamp(min=P_floor)
    return rho, P, inside


FLOORS = dict(rho_floor=1e-8, P_floor=1e-10)


def _rotating_star(n, dx, x0, gamma, seed, ghosts=True):
    rng = np.random.default_rng(seed)
    c = _centres(n, dx, x0, ghosts)
    om = float(rng.uniform(0.1, 0.3)) * math.sqrt(1.0 / 0.5 ** 3)
    X, Y, Z = c[None, None, :], c[None, :, None], c[:, None, None]
    r = torch.sqrt(X * X + Y * Y + Z * Z)
    rho, P, inside = _polytrope(r, 1.0, 1.0, 0.5, gamma, **FLOORS)
    rho = torch.where(inside, rho * (1.0 + 0.01 * _ripple(c, c, c, rng, 6.0)), rho)
    zero = torch.zeros_like(rho)
    return _pack(rho, (torch.where(inside, -om * Y + zero, zero), torch.where(inside, om * X + zero, zero), zero), P,
                 gamma)


def _exploding_star(n, dx, x0, gamma, seed):
    rng = np.random.default_rng(seed)
    c = _centres(n, dx, x0, True)
    X, Y, Z = c[None, None, :], c[None, :, None], c[:, None, None]
    r = torch.sqrt(X * X + Y * Y + Z * Z)
    rho, P, inside = _polytrope(r, 3.0, 10.0, 1.0, gamma, **FLOORS)
    rho = torch.where(inside, rho * (1.0 + 0.01 * _ripple(c, c, c, rng, 4.0)), rho)
    P = P + torch.where(r < 0.3, 0.2 * P, torch.zeros_like(P))          # the bomb
    h = float(rng.uniform(0.2, 0.6))                                    # homologous expansion
    vr = torch.where(inside, torch.full_like(rho, h), torch.zeros_like(rho))
    return _pack(rho, (vr * X, vr * Y, vr * Z), P, gamma)


def _binary(dx, seed):
    """Two black holes of mass 5 on their circular orbit of separation 3 at a seeded phase."""
    ph = float(np.random.default_rng(seed + 77).uniform(0, 2 * math.pi))
    v = math.sqrt(10.0 / 3.0) / 2.0
    p = (1.5 * math.cos(ph), 1.5 * math.sin(ph), 0.0)
    u = (-v * math.sin(ph), v * math.cos(ph), 0.0)
    return [(p, u, 5.0, 2 * dx, 1e6, 4 * dx), (tuple(-a for a in p), tuple(-a for a in u), 5.0, 2 * dx, 1e6, 4 * dx)]


def _gamma(case):
    return {"fmr": 2.0, "nested": 4.0 / 3.0, "coupled": 4.0 / 3.0}.get(case["kind"], 5.0 / 3.0)


UNIFORM = dict(rho_floor=1e-6, P_floor=1e-6)
CFL = 0.4


def _density(case, seed):
    """A clumpy density on [-1, 1]^3, the kind of field whose potential the runs solve for."""
    rng = np.random.default_rng(seed)
    n = (case["nx"], case["ny"], case["nz"])
    d = [2.0 / m for m in n]
    xc, yc, zc = (_centres(m, h, -1.0, False) for m, h in zip(n, d))
    rho = 1e-8
    for _ in range(3):
        c, w = rng.uniform(-0.4, 0.4, 3), float(rng.uniform(0.1, 0.3))
        r2 = ((xc - float(c[0])) ** 2)[None, None, :] + ((yc - float(c[1])) ** 2)[None, :, None] \
            + ((zc - float(c[2])) ** 2)[:, None, None]
        rho = rho + torch.exp(-r2 / (w * w))
    return rho.permute(2, 1, 0), d


def _levels(case, seed):
    """The mesh levels of a refined case: (level states, spacing of the base grid, boxes, lower corner)."""
    n, g = case["n"], _gamma(case)
    lo, hi = n // 4 + 1, 3 * n // 4
    box = (lo, hi, lo, hi, lo, hi, 2)
    L, nlev = (2.0, 2) if case["kind"] == "fmr" else (8.0, 3)
    fill = _rotating_star if case["kind"] == "fmr" else _exploding_star
    dx, x0, out = 2 * L / n, -L, []
    for _ in range(nlev):
        out.append(fill(n, dx, x0, g, seed))
        x0, dx = x0 + (lo - 1) * dx, dx / 2
    return out, 2 * L / n, (box,) * (nlev - 1), -L


def prepare(case, seed):
    k, S = case["kind"], {"case": case}
    if case["precision"] == "learned":
        from bsn import learned
        learned.install(*learned.load_params())
    if k in ("step", "run", "rhs"):
        n = (case["nx"], case["ny"], case["nz"])
        S["U0"], S["dx"] = _blast(*n, _gamma(case), seed)
        if k == "rhs":
            S["U"], S["dU"], S["F"] = S.pop("U0"), bsn.state(*n), bsn.flux_arrays(*n)
        else:
            S["U"] = S["U0"].clone()
    elif k == "poisson":
        S["rho"], S["d"] = _density(case, seed)
    elif k == "coupled":
        n = case["n"]
        S["dx"] = 8.0 / n
        S["U0"] = _exploding_star(n, S["dx"], -4.0, _gamma(case), seed)
        S["U"], S["bhs"] = S["U0"].clone(), _binary(S["dx"], seed)
        S["diag"] = torch.zeros((case["steps"], bsn.DIAG_RECORD), dtype=F64, device=DEV)
    else:
        init, dx, boxes, x0 = _levels(case, seed)
        n = case["n"]
        U = init[0].clone()
        if k == "fmr":
            H = bsn.FMRGrid3D(U, n, n, n, dx, *boxes[0][:6], boxes[0][6], _gamma(case), init=False, **FLOORS)
            lev, pairs = [H.Uc, H.Uf], [H]
        else:
            H = bsn.FMRHierarchy3D(U, n, n, n, dx, boxes, _gamma(case), init=False, **FLOORS)
            lev, pairs = H.levels, H.pairs
        for a, b in zip(lev, init):
            a.copy_(b)
        for p in reversed(pairs):   # every level holds the restriction of the finer ones
            p.restrict()
        S.update(H=H, lev=lev, init=[a.clone() for a in lev], x0=x0, dxf=dx / 2 ** len(boxes))
        if k == "nested":
            S["bhs"] = _binary(S["dxf"], seed)
            S["diag"] = torch.zeros((case["steps"], bsn.DIAG_RECORD), dtype=F64, device=DEV)
    return S


# ---------------------------------------------------------------------------
# one pass

def _bh_values(bhs):
    return np.array([[*b.pos, *b.vel, b.mass] for b in bhs])


def run(S):
    c = S["case"]
    k, prec, g = c["kind"], c["precision"], _gamma(c)
    if k == "step":
        n, dx, U = (c["nx"], c["ny"], c["nz"]), S["dx"], S["U"]
        U.copy_(S["U0"])
        dt = bsn.cfl_dt_3d(U, *n, dx, dx, dx, g, CFL)
        step = {"f64": bsn.euler3d_step, "f32": bsn.euler3d_step_f32, "learned": bsn.euler3d_step_learned}[prec]
        step(U, *n, dx, dx, dx, dt, g, bc=c["bc"], **UNIFORM)
        return {"U": U, "dt": dt}
    if k == "run":
        n, dx, U = (c["nx"], c["ny"], c["nz"]), S["dx"], S["U"]
        U.copy_(S["U0"])
        t, done = bsn.run_steps(U, *n, dx, dx, dx, g, CFL, n_steps=c["steps"], bc=c["bc"], precision=prec, **UNIFORM)
        return {"U": U, "t": t, "steps": done}
    if k == "rhs":
        n, dx = (c["nx"], c["ny"], c["nz"]), S["dx"]
        rhs = bsn.euler3d_rhs if prec == "f64" else bsn.euler3d_rhs_f32
        rhs(S["dU"], *S["F"], S["U"], *n, dx, dx, dx, g, bc=c["bc"], **UNIFORM)
        return {"dU": S["dU"], "F": S["F"], "U": S["U"]}
    if k == "poisson":
        return bsn.solve_poisson_isolated(S["rho"], c["nx"], c["ny"], c["nz"], *S["d"], precision=prec)
    if k == "coupled":
        n, dx, U = c["n"], S["dx"], S["U"]
        U.copy_(S["U0"])
        bhs = [bsn.BlackHole(*b) for b in S["bhs"]]
        t, done = bsn.coupled_run_steps(U, bhs, n, n, n, dx, -4.0, -4.0, -4.0, g, CFL, n_steps=c["steps"],
                                        self_gravity=c["self_gravity"], precision=prec, diag=S["diag"], **FLOORS)
        return {"U": U, "t": t, "steps": done, "bhs": _bh_values(bhs), "diag": S["diag"]}
    for a, b in zip(S["lev"], S["init"]):
        a.copy_(b)
    if k == "fmr":
        t, done = bsn.fmr3d_run_steps(S["H"], CFL, n_steps=c["steps"], precision=prec, self_gravity=c["self_gravity"])
        return {"levels": S["lev"], "t": t, "steps": done}
    bhs = [bsn.BlackHole(*b) for b in S["bhs"]]
    t, done = bsn.coupled_nested_run_steps(S["H"], bhs, S["x0"], S["x0"], S["x0"], CFL, n_steps=c["steps"],
                                           self_gravity=c["self_gravity"], precision=prec, diag=S["diag"])
    return {"levels": S["lev"], "t": t, "steps": done, "bhs": _bh_values(bhs), "diag": S["diag"]}


def _poisson_work(nx, ny, nz):
    N = 8 * nx * ny * nz
    return dict(bytes=16.0 * nx * ny * nz, flops=2 * 2.5 * N * math.log2(N))


def work(case):
    """State read once and written once per step, the scheme's operations per
    cell and step (a refined level counts once per subcycle), and the padded
    transforms of each Poisson solve."""
    k = case["kind"]
    if k == "poisson":
        return _poisson_work(case["nx"], case["ny"], case["nz"])
    if k in ("step", "run", "rhs"):
        cells = case["nx"] * case["ny"] * case["nz"]
        if k == "rhs":   # a third of a step; the state in, the right-hand side and three flux arrays out
            return dict(bytes=5 * 40.0 * cells, flops=FLOPS_PER_CELL_STEP / 3 * cells)
        s = case.get("steps", 1)
        return dict(bytes=80.0 * cells * s, flops=FLOPS_PER_CELL_STEP * cells * s)
    n3, s = float(case["n"]) ** 3, case["steps"]
    units, levels, solves = {"coupled": (1, 1, 3), "fmr": (3, 2, 1), "nested": (7, 3, 1)}[k]
    w = dict(bytes=80.0 * levels * n3 * s, flops=FLOPS_PER_CELL_STEP * units * n3 * s)
    if case["self_gravity"]:
        w["flops"] += s * solves * _poisson_work(case["n"], case["n"], case["n"])["flops"]
    return w


# ---------------------------------------------------------------------------
# the uniform-grid paths in plain torch, 64 bits.  A state is (5, Z, Y, X).

def _sh(a, axis, lo, n):
    return a.narrow(a.dim() - 1 - axis, lo, n)


def _weno_weights(b0, b1, b2, d):
    tau = (b0 - b2).abs()
    a = [dk * (1 + (tau / (1e-36 + b)) ** 2) for dk, b in zip(d, (b0, b1, b2))]
    s = a[0] + a[1] + a[2]
    return [x / s for x in a]


def _indicators(v, side):
    k = 13 / 12
    b0 = k * (v[0] - 2 * v[1] + v[2]) ** 2
    b1 = k * (v[1] - 2 * v[2] + v[3]) ** 2
    b2 = k * (v[2] - 2 * v[3] + v[4]) ** 2 + 0.25 * (3 * v[2] - 4 * v[3] + v[4]) ** 2
    if side == 0:
        return b0 + 0.25 * (v[0] - 4 * v[1] + 3 * v[2]) ** 2, b1 + 0.25 * (v[1] - v[3]) ** 2, b2
    return b0 + 0.25 * (v[0] - v[2]) ** 2, b1 + 0.25 * (v[1] - 4 * v[2] + 3 * v[3]) ** 2, b2


def _net_weights(u, P):
    """The 5-32-32-3 network's softmax weights of normalised stencils u (n, 5)."""
    W1, b1, W2, b2, W3, b3 = P
    h = torch.relu(u @ W1.T + b1)
    h = torch.relu(h @ W2.T + b2)
    return torch.softmax(h @ W3.T + b3, dim=1)


def _reconstruct(v, side, net):
    b = _indicators(v, side)
    d = (0.1, 0.6, 0.3) if side == 0 else (0.3, 0.6, 0.1)
    w = _weno_weights(*b, d)
    if net is not None:
        c = v[2] if side == 0 else v[1]
        spread = (v[0] - c).abs()
        for x in v[1:]:
            spread = torch.maximum(spread, (x - c).abs())
        bmin = torch.minimum(torch.minimum(b[0], b[1]), b[2])
        use = ((b[0] - b[2]).abs() <= 4 * (bmin + 1e-3 * spread ** 2)) & (spread > 1e-15) & (spread > 1e-6 * c.abs())
        at = use.nonzero(as_tuple=True)
        if at[0].numel():
            u = torch.stack([(x[at] - c[at]) / spread[at] for x in v], 1)
            wn = _net_weights(u, net[side])
            for i in range(3):
                w[i][at] = wn[:, i]
    if side == 0:
        q = (v[0] / 3 - 7 / 6 * v[1] + 11 / 6 * v[2], -v[1] / 6 + 5 / 6 * v[2] + v[3] / 3,
             v[2] / 3 + 5 / 6 * v[3] - v[4] / 6)
    else:
        q = (-v[0] / 6 + 5 / 6 * v[1] + v[2] / 3, v[1] / 3 + 5 / 6 * v[2] - v[3] / 6,
             11 / 6 * v[2] - 7 / 6 * v[3] + v[4] / 3)
    return w[0] * q[0] + w[1] * q[1] + w[2] * q[2]


def _hllc(L, R, ax, g):
    one = torch.ones_like(L[0])

    def side(W):
        r, m, E = W[0], [W[1 + ax], W[1 + (ax + 1) % 3], W[1 + (ax + 2) % 3]], W[4]
        ok = r > 0
        r = torch.where(ok, r.clamp(min=1e-30), 1e-30 * one)
        m = [torch.where(ok, x, 0 * one) for x in m]
        E = torch.where(ok, E, 0 * one)
        m2 = m[0] ** 2 + m[1] ** 2 + m[2] ** 2
        s = torch.where(m2 > r * r * 1e4, r * 100 / m2.clamp(min=1e-300).sqrt(), one)
        m = [x * s for x in m]
        KE = torch.minimum(0.5 * (m[0] ** 2 + m[1] ** 2 + m[2] ** 2) / r, 0.5 * r * 1e4)
        E = torch.maximum(E, KE)
        p = (g - 1) * (E - KE)
        v = [x / r for x in m]
        F = [m[0], r * v[0] ** 2 + p, m[1] * v[0], m[2] * v[0], (E + p) * v[0]]
        return r, m, E, p, v, (g * p / r).sqrt(), F

    rL, mL, EL, pL, vL, cL, FL = side(L)
    rR, mR, ER, pR, vR, cR, FR = side(R)
    ps = (0.5 * (pL + pR) - 0.5 * (vR[0] - vL[0]) * 0.5 * (rL + rR) * 0.5 * (cL + cR)).clamp(min=0)
    gg = (g + 1) / (2 * g)

    def q(p):
        return torch.where(ps > p, (1 + gg * (ps / p.clamp(min=1e-300) - 1)).clamp(min=0).sqrt(), one)

    both = (pL > 0) & (pR > 0)
    SL = torch.where(both, vL[0] - cL * q(pL), torch.minimum(vL[0] - cL, vR[0] - cR))
    SR = torch.where(both, vR[0] + cR * q(pR), torch.maximum(vL[0] + cL, vR[0] + cR))
    den = rL * (SL - vL[0]) - rR * (SR - vR[0])
    S = (pR - pL + mL[0] * (SL - vL[0]) - mR[0] * (SR - vR[0])) / torch.where(den == 0, one, den)
    UL, UR = [rL, *mL, EL], [rR, *mR, ER]

    def star(r, m, E, p, v, F, Sk, U):
        d = r * (Sk - v[0])
        chi = d / (Sk - S)
        Es = torch.where(d.abs() > 1e-100, chi * (E / r + (S - v[0]) * (S + p / d)), 0 * one)
        X = [chi, chi * S, chi * v[1], chi * v[2], Es]
        return [f + Sk * (x - u) for f, x, u in zip(F, X, U)]

    sl, sr = star(rL, mL, EL, pL, vL, FL, SL, UL), star(rR, mR, ER, pR, vR, FR, SR, UR)
    steep = torch.maximum(rL, rR) > 3 * torch.minimum(rL, rR)
    out = []
    for i in range(5):
        hll = (SR * FL[i] - SL * FR[i] + SL * SR * (UR[i] - UL[i])) / (SR - SL)
        f = torch.where(steep, hll, torch.where(S >= 0, sl[i], sr[i]))
        f = torch.where(SL >= 0, FL[i], torch.where(SR <= 0, FR[i], f))
        out.append(torch.where(den.abs() < 1e-100, 0 * one, f))
    back = {1 + ax: out[1], 1 + (ax + 1) % 3: out[2], 1 + (ax + 2) % 3: out[3]}
    return torch.stack([out[0], back[1], back[2], back[3], out[4]])


def _act(a):
    return a[..., NG:-NG, NG:-NG, NG:-NG]


def _fill(U, bc):
    for ax in range(3):
        n = U.shape[3 - ax] - 2 * NG
        for t in range(NG):
            lo, hi = (NG, NG + n - 1) if bc == "outflow" else (n + t, NG + t)
            U.narrow(3 - ax, t, 1).copy_(U.narrow(3 - ax, lo, 1))
            U.narrow(3 - ax, NG + n + t, 1).copy_(U.narrow(3 - ax, hi, 1))


def _floor(U, g, rho_floor, P_floor):
    A = _act(U)
    low = A[0] < rho_floor
    KE = 0.5 * (A[1] ** 2 + A[2] ** 2 + A[3] ** 2) / torch.where(low, torch.ones_like(A[0]), A[0])
    E = torch.where((g - 1) * (A[4] - KE) < P_floor, P_floor / (g - 1) + KE, A[4])
    A[4] = torch.where(low, torch.full_like(E, P_floor / (g - 1)), E)
    for q in (1, 2, 3):
        A[q][low] = 0.0
    A[0][low] = rho_floor


def _fluxes(U, g, ax, net):
    """Fluxes of every interface along one axis between active cells, (5, ...) with one more along it."""
    n = [U.shape[3 - a] - 2 * NG for a in range(3)]
    r = U[0].clamp(min=1e-30)
    P = ((g - 1) * (U[4] - 0.5 * (U[1] ** 2 + U[2] ** 2 + U[3] ** 2) / r)).clamp(min=0)

    def cells(a):
        for b in range(3):
            if b != ax:
                a = _sh(a, b, NG, n[b])
        return [_sh(a, ax, s, n[ax] + 1) for s in range(6)]

    L, R = [], []
    for a in (U[0], U[1], U[2], U[3], P):
        v = cells(a)
        L.append(_reconstruct(v[:5], 0, net))
        R.append(_reconstruct(v[1:], 1, net))
    p = cells(P)
    for W, st in ((L, p[:5]), (R, p[1:])):
        top = st[0]
        for x in st[1:]:
            top = torch.maximum(top, x)
        W[4] = torch.minimum(W[4].clamp(min=0), top)
        rp = W[0].clamp(min=1e-30)
        W[4] = W[4] / (g - 1) + torch.minimum(0.5 * (W[1] ** 2 + W[2] ** 2 + W[3] ** 2) / rp, 0.5 * rp * 1e4)
    return _hllc(L, R, ax, g)


def _rhs(U, dx, g, bc, floors, net=None, keep=None):
    """Ghosts and floors of U, then the flux divergence over the active cells."""
    _fill(U, bc)
    _floor(U, g, **floors)
    d = 0.0
    for ax in range(3):
        F = _fluxes(U, g, ax, net)
        n = F.shape[3 - ax] - 1
        d = d - (_sh(F, ax, 1, n) - _sh(F, ax, 0, n)) / dx
        if keep is not None:
            keep.append(F)
    return d


def _step(U, dt, dx, g, bc, floors, net=None, source=None):
    Un = U.clone()
    for a, b, c in ((1.0, 0.0, 1.0), (0.75, 0.25, 0.25), (1 / 3, 2 / 3, 2 / 3)):
        d = _rhs(U, dx, g, bc, floors, net)
        if source is not None:
            source(_act(U), d)
        if b == 0.0:
            U.copy_(Un)
        else:
            U.mul_(b).add_(Un, alpha=a)
        _act(U).add_(d, alpha=c * dt)
        _floor(U, g, **floors)


def _speed(U, dx, g):
    A = _act(U)
    r = A[0].clamp(min=1e-30)
    v = [A[q] / r for q in (1, 2, 3)]
    P = ((g - 1) * (A[4] / r - 0.5 * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)) * r).clamp(min=0)
    c = (g * P / r).sqrt()
    return float(max((x.abs() + c).max() for x in v)) / dx


def _potential(rho, d):
    n = rho.shape[::-1]
    r2 = 0.0
    for ax, (m, h) in enumerate(zip(n, d)):
        i = torch.arange(2 * m, device=rho.device, dtype=F64)
        i = torch.where(i < m, i, i - 2 * m) * h
        r2 = r2 + (i * i).reshape([-1 if 2 - ax == b else 1 for b in range(3)])
    dV = d[0] * d[1] * d[2]
    K = torch.fft.rfftn(-1.0 / torch.sqrt(r2 + dV ** (2 / 3)))
    s = tuple(2 * m for m in rho.shape)
    phi = torch.fft.irfftn(torch.fft.rfftn(rho, s=s) * K, s=s)
    return dV * phi[:n[2], :n[1], :n[0]]


def _gravity(A, d, phi, dx):
    v = 0.0
    for ax in range(3):
        n = phi.shape[2 - ax]
        i = torch.arange(n, device=phi.device)
        hi, lo = (i + 1).clamp(max=n - 1), (i - 1).clamp(min=0)
        w = ((hi - lo).to(F64) * dx).reshape([-1 if 2 - ax == b else 1 for b in range(3)])
        gr = (phi.index_select(2 - ax, hi) - phi.index_select(2 - ax, lo)) / w
        d[1 + ax] -= A[0] * gr
        v = v + A[1 + ax] * gr
    d[4] -= v


def _network(case):
    if case["precision"] != "learned":
        return None
    z = np.load(os.path.join(os.getcwd(), "binary-supernova_b200", "bsn", "weno_mlp.npz"))
    out = []
    for key in ("left", "right"):
        p = torch.as_tensor(z[key], device=DEV, dtype=F64)
        cut = (160, 32, 1024, 32, 96, 3)
        a = torch.split(p, cut)
        out.append((a[0].reshape(32, 5), a[1], a[2].reshape(32, 32), a[3], a[4].reshape(3, 32), a[5]))
    return out


def _plain(U):
    return U.permute(0, 3, 2, 1).contiguous()


def _exact_coupled(case, seed):
    n, g, dx, x0 = case["n"], _gamma(case), 8.0 / case["n"], -4.0
    U = _plain(_exploding_star(n, dx, x0, g, seed))
    c = _centres(n, dx, x0, False)
    xyz = (c[None, None, :], c[None, :, None], c[:, None, None])
    bh = [dict(p=np.array(p), v=np.array(v), m=m, eps=e, rs=max(6 * m / cc ** 2, rf)) for p, v, m, e, cc, rf in
          _binary(dx, seed)]

    def offsets(b):
        return [x - float(p) for x, p in zip(xyz, b["p"])]

    def t_sink(b):
        return b["rs"] / math.sqrt(2 * b["m"] / b["rs"])

    def source(A, d):
        acc = [0.0, 0.0, 0.0]
        for b in bh:
            o = offsets(b)
            r2 = o[0] ** 2 + o[1] ** 2 + o[2] ** 2 + b["eps"] ** 2
            acc = [a - b["m"] / (r2 * r2.sqrt()) * x for a, x in zip(acc, o)]
        for q in range(3):
            d[1 + q] += A[0] * acc[q]
            d[4] += A[1 + q] * acc[q]
        if case["self_gravity"]:
            _gravity(A, d, _potential(A[0].contiguous(), (dx, dx, dx)), dx)
        for b in bh:
            o = offsets(b)
            rr = (o[0] ** 2 + o[1] ** 2 + o[2] ** 2).sqrt()
            inside = (rr < b["rs"]) & (A[0] > 0)
            w = torch.where(inside, torch.full_like(rr, 1 / t_sink(b)), torch.zeros_like(rr))
            v = [A[1 + q] / A[0] for q in range(3)]
            n_ = [x / rr for x in o]
            vr = sum((v[q] - float(b["v"][q])) * n_[q] for q in range(3))
            e = A[4] / A[0] - 0.5 * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
            d[0] -= A[0] * w
            for q in range(3):
                d[1 + q] -= A[0] * vr * n_[q] * w
            d[4] -= (0.5 * A[0] * vr ** 2 + A[0] * e) * w

    def accel(F):
        out = []
        for i, b in enumerate(bh):
            a = F[i] / b["m"]
            for j, o in enumerate(bh):
                if j != i:
                    x = o["p"] - b["p"]
                    r2 = float(x @ x) + o["eps"] ** 2
                    a = a + o["m"] / (r2 * math.sqrt(r2)) * x
            out.append(a)
        return out

    t = 0.0
    for _ in range(case["steps"]):
        dt = CFL / _speed(U, dx, g)
        A, F = _act(U), []
        for b in bh:
            o = offsets(b)
            r2 = o[0] ** 2 + o[1] ** 2 + o[2] ** 2 + b["eps"] ** 2
            w = b["m"] / (r2 * r2.sqrt()) * A[0] * dx ** 3
            f = np.array([float((w * x).sum()) for x in o])
            F.append(f if np.isfinite(f).all() and np.linalg.norm(f) <= 1e3 else 0 * f)
        p0, v0 = [b["p"] for b in bh], [b["v"] for b in bh]
        for a_, b_ in ((0.0, 1.0), (0.75, 0.25), (1 / 3, 2 / 3)):
            dv = accel(F)
            for i, b in enumerate(bh):
                p, v = b["p"] + dt * b["v"], b["v"] + dt * dv[i]
                b["p"], b["v"] = a_ * p0[i] + b_ * p, a_ * v0[i] + b_ * v
        _step(U, dt, dx, g, "outflow", FLOORS, _network(case), source)
        A = _act(U)
        for b in bh:
            o = offsets(b)
            inside = ((o[0] ** 2 + o[1] ** 2 + o[2] ** 2).sqrt() < b["rs"]) & (A[0] > 0)
            rate = dx ** 3 / t_sink(b) * dt
            dm = float(A[0][inside].sum()) * rate
            if dm > 0:
                dp = np.array([float(A[q][inside].sum()) for q in (1, 2, 3)]) * rate
                b["v"] = (b["m"] * b["v"] + dp) / (b["m"] + dm)
                b["m"] += dm
                b["rs"] = max(6 * b["m"] / 1e12, 4 * dx)
        t += dt
    out = np.array([[*b["p"], *b["v"], b["m"]] for b in bh])
    return {"U": U.permute(0, 3, 2, 1), "t": t, "steps": case["steps"], "bhs": out, "diag": None}


def exact(case, seed):
    k, g = case["kind"], _gamma(case)
    if k in ("fmr", "nested"):   # whole runs on several levels: no restatement
        return None
    if k == "coupled":
        return _exact_coupled(case, seed)
    if k == "poisson":
        rho, d = _density(case, seed)
        return _potential(rho.permute(2, 1, 0).contiguous(), d).permute(2, 1, 0)
    U, dx = _blast(case["nx"], case["ny"], case["nz"], g, seed)
    U, net = _plain(U), _network(case)
    if k == "rhs":
        F, out = [], []
        d = _rhs(U, dx, g, case["bc"], UNIFORM, keep=F)
        dU = torch.zeros_like(U)
        _act(dU).copy_(d)
        for ax, f in enumerate(F):   # the reference's flux arrays: one longer along their axis
            shape = list(U.shape)
            shape[3 - ax] += 1
            full = torch.zeros(shape, device=U.device, dtype=F64)
            v = full
            for a in range(3):
                v = v.narrow(3 - a, NG - (a == ax), f.shape[3 - a])
            # face i of the array lies above cell i
            v.copy_(f)
            out.append(full.permute(0, 3, 2, 1))
        return {"dU": dU.permute(0, 3, 2, 1), "F": out, "U": U.permute(0, 3, 2, 1)}
    if k == "step":
        dt = CFL / _speed(U, dx, g)
        _step(U, dt, dx, g, case["bc"], UNIFORM, net)
        return {"U": U.permute(0, 3, 2, 1), "dt": dt}
    t = 0.0
    for _ in range(case["steps"]):
        dt = CFL / _speed(U, dx, g)
        _step(U, dt, dx, g, case["bc"], UNIFORM, net)
        t += dt
    return {"U": U.permute(0, 3, 2, 1), "t": t, "steps": case["steps"]}
