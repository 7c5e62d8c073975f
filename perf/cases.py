"""Timed cases of the SD-ADER step, through the package's public entry points.

Every case is a simulation as a user runs it: a simulator is built once, holds its
buffers, and is then given states to advance.  ``api`` says through which door:

* ``host``: ``perform_iterations`` on states assigned to ``sim.dm`` and read back from it
  as NumPy arrays (the class surface of the reference);
* ``device``: ``adjoint.run_steps`` on a CUDA tensor (states that stay on the GPU);
* ``gradient``: ``run_steps`` and its backward pass;
* ``ensemble``: ``SDADER_Ensemble.perform_iterations`` over simulators of several sizes.

Sizes, problems and options are those of the package's benchmark, tests and problem
library, with odd sizes among them.
"""
import math

import numpy as np
import torch

from spd_gb300 import SDADER_Ensemble, SDADER_Simulator
from spd_gb300.adjoint import run_steps

GAMMA = 1.4
CFL = 0.8
MIN_C2 = 1e-10
TOL = 1e-5          # relative tolerance of the discrete maximum principle
MIN_RHO, MAX_RHO, MIN_P = 1e-10, 1e10, 1e-10
NU, BETA = 1e-3, 2.0 / 3
GRAVITY = 1.0
SIDES = (16, 24, 32, 48, 64)
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"

# what a problem fixes: box length per direction, boundary kind
PROBLEMS = {
    "wave": dict(box=1.0, bc="periodic"),        # density wave carried by a uniform flow
    "step": dict(box=1.0, bc="periodic"),        # the same with a density box: troubled cells
    "vortex": dict(box=10.0, bc="periodic"),     # isentropic vortex
    "shear": dict(box=1.0, bc="periodic"),       # Kelvin-Helmholtz shear layer
    "quadrant": dict(box=1.0, bc="gradfree"),    # four-quadrant Riemann problem
    "blast": dict(box=1.0, bc="reflective"),     # Sedov blast
    "column": dict(box=1.0, bc="reflective"),    # atmosphere in a gravity potential
}


def _case(name, api, problem, cells, p, steps, update="FV", solver="hllc", slopes="minmod", viscous=False,
          fma=False, members=0):
    nx, ny, nz = (tuple(cells) + (0, 0))[:3]
    c = dict(api=api, problem=problem, nx=nx, ny=ny, nz=nz, p=p, steps=steps, update=update, solver=solver,
             slopes=slopes, viscous=viscous, fma=fma, members=members)
    return c if name is None else dict(name=name, **c)


def listed():
    return [
        # the reference's own 1D demonstration: launches and host calls are all there is
        _case("step_1d_64", "host", "step", (64,), 3, 10, solver="llf"),
        # the smallest 2D configuration of the benchmark, run as its users run it
        _case("vortex_32", "host", "vortex", (32, 32), 3, 10, solver="llf"),
        # the headline benchmark: shocks, limiting on, the largest 2D grid
        _case("quadrant_512", "device", "quadrant", (512, 512), 3, 1),
        # 3D blast with limiting, the benchmark's degree
        _case("blast_48", "device", "blast", (48, 48, 48), 2, 1),
        # smooth flow without limiter, a grid of odd sides (1/h no power of two)
        _case("vortex_sd_251x190", "device", "vortex", (251, 190), 3, 2, update="SD", solver="llf"),
        # low-Mach solver and moncen slopes, an odd number of subcell updates per step
        _case("shear_lhllc_150x130", "device", "shear", (150, 130), 2, 3, solver="lhllc", slopes="moncen"),
        # many small problems in one graph
        _case("ensemble_12", "ensemble", "shear", (0,), 3, 4, members=12),
        # gradient of a run with respect to its initial state
        _case("gradient_96", "gradient", "shear", (96, 96), 3, 3),
        # viscous shear layer
        _case("viscous_128", "device", "shear", (128, 128), 3, 2, update="SD", viscous=True),
        # gravity, limiting, walls, a grid longer than wide
        _case("column_96x160", "device", "column", (96, 160), 2, 2),
        # the opt-in build with fused multiply-adds
        _case("vortex_fma_200", "device", "vortex", (200, 200), 3, 2, solver="llf", fma=True),
        # the highest degree, in 3D
        _case("wave_3d_p4", "device", "wave", (21, 20, 19), 4, 1, update="SD"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("host", "plane", "plane", "smooth", "space", "viscous", "gravity", "fma", "gradient", "ensemble"))
    solver = rng.choice(("llf", "hllc", "lhllc"))
    slopes = rng.choice(("minmod", "moncen"))
    p = rng.choice((1, 2, 3, 3, 4))
    if kind == "host":
        if rng.random() < 0.5:
            return _case(None, "host", "step", (_log_int(rng, 32, 4096),), p, rng.randint(2, 12), solver=solver, slopes=slopes)
        n = _log_int(rng, 12, 96)
        return _case(None, "host", "vortex", (n, n + rng.randint(0, 5)), p, rng.randint(2, 8), solver=solver, slopes=slopes)
    if kind == "space":
        p = rng.choice((1, 2, 3, 4))
        n = _log_int(rng, 8, {3: 28, 4: 14}.get(p, 44))
        problem = rng.choice(("blast", "wave"))
        return _case(None, "device", problem, (n, n + rng.randint(0, 3), n + rng.randint(0, 3)), p, 1, solver="hllc",
                     update="FV" if problem == "blast" else rng.choice(("FV", "SD")))
    if kind == "gradient":
        n = _log_int(rng, 16, 80)
        return _case(None, "gradient", "shear", (n, n + rng.randint(0, 7)), rng.choice((1, 2, 3)), rng.randint(2, 3))
    if kind == "ensemble":
        return _case(None, "ensemble", "shear", (0,), rng.choice((2, 3)), rng.randint(1, 4), members=rng.randint(4, 16))
    nx = _log_int(rng, 40, 400 if p < 4 else 240)
    ny = max(24, int(nx * rng.uniform(0.5, 1.0)))
    if kind == "smooth":
        return _case(None, "device", "vortex", (nx, ny), p, 1, update="SD", solver=solver)
    if kind == "viscous":
        return _case(None, "device", "shear", (min(nx, 200), min(ny, 200)), p, rng.randint(1, 2), update="SD",
                     solver=rng.choice(("llf", "hllc")), viscous=True)
    if kind == "gravity":
        return _case(None, "device", "column", (min(nx, 160), min(ny, 160)), p, 1, slopes=slopes)
    if kind == "fma":
        return _case(None, "device", "vortex", (min(nx, 300), min(ny, 300)), p, 1, solver=solver, fma=True)
    return _case(None, "device", rng.choice(("quadrant", "shear")), (nx, ny), p, 1, solver=solver, slopes=slopes)


# ---------------------------------------------------------------------------
# problems: pointwise primitives f(xyz, var), var 0 density, 1..d velocities,
# d + 1 pressure, -1 the gravity potential
# ---------------------------------------------------------------------------
def _problem(case, seed, cells):
    r = np.random.default_rng(seed)
    d = len(cells)
    kind = case["problem"]

    if kind in ("wave", "step"):
        vel = r.uniform(0.5, 1.0, d)
        shift = r.uniform(0.0, 1.0, d)

        def f(x, v):
            if v == 0 and kind == "wave":
                return 1.0 + 0.125 * np.sin(2 * np.pi * sum(x[i] - shift[i] for i in range(d)))
            if v == 0:
                inside = np.ones(x[0].shape, dtype=bool)
                for i in range(d):
                    inside &= np.abs((x[i] - shift[i]) % 1.0 - 0.5) < 0.25
                return np.where(inside, 2.0, 1.0)
            return (vel[v - 1] if v <= d else 1.0) * np.ones(x[0].shape)
    elif kind == "vortex":
        cx, cy = r.uniform(4.0, 6.0, 2)
        ux, uy = r.uniform(0.7, 1.2, 2)
        beta = r.uniform(4.0, 5.5)

        def f(x, v):
            a = (x[0] - cx + 5.0) % 10.0 - 5.0
            b = (x[1] - cy + 5.0) % 10.0 - 5.0
            r2 = a * a + b * b
            T = 1.0 - (GAMMA - 1) * beta ** 2 / (8 * GAMMA * np.pi ** 2) * np.exp(1 - r2)
            du = beta / (2 * np.pi) * np.exp((1 - r2) / 2)
            if v == 0:
                return T ** (1 / (GAMMA - 1))
            return (ux - du * b) if v == 1 else (uy + du * a) if v == 2 else T ** (GAMMA / (GAMMA - 1))
    elif kind == "shear":
        table = r.normal(0.0, 1e-3, size=cells[::-1])
        rho = 2.0 + r.uniform(-0.1, 0.1)
        phase = r.uniform(0.0, 1.0, (4, 2))

        def f(x, v):
            inner = np.abs(x[1] - 0.5) < 0.25
            a, b = (2 * np.pi * (x[i] + phase[v, i]) for i in range(2))
            wave = 0.01 * np.sin(a) * np.cos(2 * b)
            if v == 0:
                return np.where(inner, rho, 1.0) * (1.0 + wave)
            if v == 1:
                return np.where(inner, 0.5, -0.5) + wave
            if v == 2:
                i = np.clip(np.floor(x[0] * cells[0]).astype(np.int64), 0, cells[0] - 1)
                j = np.clip(np.floor(x[1] * cells[1]).astype(np.int64), 0, cells[1] - 1)
                return wave + table[j, i]
            return 2.5 * (1.0 + wave)
    elif kind == "quadrant":
        s = 1.0 + r.uniform(-0.02, 0.02, 4)
        x0, y0 = (round(n * r.uniform(0.45, 0.55)) / n for n in cells)
        table = ((1.5 * s[0], 0.5323 * s[1], 0.138 * s[2], 0.5323 * s[3]), (0.0, 1.206, 1.206, 0.0),
                 (0.0, 0.0, 1.206, 1.206), (1.5, 0.3, 0.029, 0.3))

        def f(x, v):
            ur, ul, ll, lr = table[v]
            return np.where(x[0] >= x0, np.where(x[1] >= y0, ur, lr), np.where(x[1] >= y0, ul, ll))
    elif kind == "blast":
        h = [1.0 / n for n in cells]
        rho = 1.0 + r.uniform(-0.05, 0.05)
        at = [round(n * r.uniform(0.4, 0.6)) / n for n in cells]
        hot = (GAMMA - 1) / (8 * h[0] * h[1] * h[2])

        def f(x, v):
            if v == 0:
                return rho * np.ones(x[0].shape)
            if v == d + 1:
                inside = np.ones(x[0].shape, dtype=bool)
                for i in range(d):
                    inside &= np.abs(x[i] - at[i]) < h[i]
                return np.where(inside, hot, 1e-5)
            return np.zeros(x[0].shape)
    else:  # column
        amp, phase = r.uniform(0.005, 0.02), r.uniform(0.0, 1.0)

        def f(x, v):
            z = x[d - 1]
            if v == -1:
                return GRAVITY * z
            if v == 0:
                return np.exp(-GRAVITY * z) * (1.0 + amp * np.sign(np.sin(2 * np.pi * (x[0] - phase))))
            return np.exp(-GRAVITY * z) if v == d + 1 else np.zeros(z.shape)
    return f


def _members(case, seed):
    """(cells, seed) of every simulation of a case."""
    if case["api"] == "ensemble":
        r = np.random.default_rng(1000 + case["members"])
        return [((int(s), int(s)), seed + 7919 * i) for i, s in enumerate(r.choice(SIDES, case["members"]))]
    return [(tuple(n for n in (case["nx"], case["ny"], case["nz"]) if n), seed)]


def _solution_points(p):
    return 0.5 * (1.0 - np.cos((2 * np.arange(p + 1) + 1) / (2 * (p + 1)) * np.pi))


def _initial(case, cells, seed):
    """Conservative state at the solution points, (V, [Nz,] [Ny,] Nx, [nz,] [ny,] nx)."""
    d, box, x = len(cells), PROBLEMS[case["problem"]]["box"], _solution_points(case["p"])
    f = _problem(case, seed, cells)
    grids = []
    for i in range(d):
        shape = [1] * (2 * d)
        shape[d - 1 - i], shape[2 * d - 1 - i] = cells[i], case["p"] + 1
        grids.append(((np.arange(cells[i])[:, None] + x) * (box / cells[i])).reshape(shape))
    xyz = np.stack(np.broadcast_arrays(*grids))
    W = np.stack([f(xyz, v) for v in range(d + 2)])
    U = W.copy()
    U[1:d + 1] *= W[0]
    U[d + 1] = W[d + 1] / (GAMMA - 1) + 0.5 * W[0] * (W[1:d + 1] ** 2).sum(0)
    return U


def prepare(case, seed):
    sims, states = [], []
    for cells, s in _members(case, seed):
        d, box, bc = len(cells), PROBLEMS[case["problem"]]["box"], PROBLEMS[case["problem"]]["bc"]
        lims = {k: (0, box) for k in ("xlim", "ylim", "zlim")[:d]}
        sims.append(SDADER_Simulator(
            p=case["p"], N=cells, init_fct=_problem(case, s, cells), update=case["update"], FB=case["update"] == "FV",
            riemann_solver_sd=case["solver"], riemann_solver_fv=case["solver"], slope_limiter=case["slopes"],
            BC=((bc, bc),) * d, cfl_coeff=CFL, viscosity=case["viscous"], nu=NU, beta=BETA,
            potential=case["problem"] == "column", fma=case["fma"], **lims))
        states.append(_initial(case, cells, s))
    state = dict(case=case, sims=sims, steps=case["steps"])
    if case["api"] in ("host", "ensemble"):
        # what such a program assigns: the solution and the primitives of its cell means
        ops = _operators(case["p"])
        state["U"] = states
        state["W"] = [_np(_prim(_means(ops, _t(U)))) for U in states]
    else:
        state["U"] = [_t(U) for U in states]
    if case["api"] == "ensemble":
        state["ensemble"] = SDADER_Ensemble(sims)
    if case["api"] == "gradient":
        g = torch.Generator(device=DEVICE).manual_seed(int(seed))
        state["dy"] = torch.randn(state["U"][0].shape, dtype=torch.float64, device=DEVICE, generator=g)
        state["U"][0].requires_grad_(True)
    return state


def run(state):
    api, sims = state["case"]["api"], state["sims"]
    if api == "device":
        return run_steps(sims[0], state["U"][0], state["steps"])
    if api == "gradient":
        U = state["U"][0]
        out = run_steps(sims[0], U, state["steps"])
        (grad,) = torch.autograd.grad(out, U, state["dy"])
        return {"U": out.detach(), "grad": grad}
    for sim, U, W in zip(sims, state["U"], state["W"]):
        sim.dm.U_sp = U
        sim.dm.W_cv = W
    if api == "ensemble":
        state["ensemble"].perform_iterations(state["steps"])
        return [sim.dm.U_sp for sim in sims]
    sims[0].perform_iterations(state["steps"])
    return {"U": sims[0].dm.U_sp, "W": sims[0].dm.W_cv}


def work(case):
    """One read of every given state and one write of every result; the operations of the
    scheme (interpolation, fluxes, Riemann problems, derivative, Picard update, subcell
    update), a divide or root counted as one."""
    total, flops = 0.0, 0.0
    p, m = case["p"], case["p"]
    n, nf, T = p + 1, p + 2, m + 1
    for cells, _ in _members(case, 0):
        d = len(cells)
        V, nc, ns = d + 2, math.prod(cells), n ** d
        sweeps = 1 + m * T                                   # (iteration, node) pairs evaluated
        lines = d * ns // n
        per = sweeps * lines * V * nf * (2 * n - 1)          # solution to flux points
        per += sweeps * lines * (nf - 2) * (6 * d + 14)      # primitives and fluxes
        per += sweeps * lines * (80 if case["solver"] == "llf" else 90)
        per += (sweeps - (T if case["update"] == "FV" else 0)) * d * V * ns * 2 * nf
        per += m * V * ns * T * (2 * T + 1)
        if case["viscous"]:
            per += sweeps * lines * nf * (2 * n * V * d + 2 * V * d + 20 * d)
        if case["update"] == "FV":
            per += 2 * V * ns * (2 * ns - 1) + T * lines * nf * V * (2 * n - 1) * (d - 1)
            per += T * ns * (V * (3 * d + 2) + 12 + 6 * d + V * (2 * d + 4))
        times = case["steps"] * (4.0 if case["api"] == "gradient" else 1.0)
        flops += per * nc * times
        arrays = {"host": 4, "device": 2, "ensemble": 3, "gradient": 4}[case["api"]]
        total += 8.0 * V * ns * nc * arrays
    return {"bytes": total, "flops": flops}


# ---------------------------------------------------------------------------
# the same steps in plain 64-bit torch
# ---------------------------------------------------------------------------
def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=DEVICE)


def _np(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _lagrange(to, frm):
    out = np.ones((len(to), len(frm)))
    for i in range(len(frm)):
        for k in range(len(frm)):
            if k != i:
                out[:, i] *= (to - frm[k]) / (frm[i] - frm[k])
    return out


def _lagrange_prime(to, frm):
    out = np.zeros((len(to), len(frm)))
    for i in range(len(frm)):
        for j in range(len(frm)):
            if j == i:
                continue
            term = np.full(len(to), 1.0 / (frm[i] - frm[j]))
            for k in range(len(frm)):
                if k not in (i, j):
                    term = term * (to - frm[k]) / (frm[i] - frm[k])
            out[:, i] += term
    return out


def _legendre(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (x + 1.0), 0.5 * w


def _operators(p):
    sp = _solution_points(p)
    fp = np.hstack((0.0, _legendre(p)[0], 1.0))
    q, wq = _legendre(p)
    means = np.stack([wq @ _lagrange(fp[i] + (fp[i + 1] - fp[i]) * q, sp) for i in range(p + 1)])
    tp, wt = _legendre(p + 1)
    end = _lagrange(np.array([1.0]), tp)[0]
    ader = np.outer(end, end) - _lagrange_prime(tp, tp).T * wt
    return dict(fp=fp, interp=_t(_lagrange(fp, sp)), deriv=_t(_lagrange_prime(sp, fp)), means=_t(means),
                points=_t(np.linalg.inv(means)), picard=_t(np.linalg.inv(ader) * wt), weights=wt)


def _along(A, M, axis):
    return torch.movedim(torch.movedim(M, axis, -1) @ A.T, -1, axis)


def _means(ops, U):
    d = (U.dim() - 1) // 2
    for i in range(d):
        U = _along(ops["means"], U, -1 - i)
    return U


def _cut(M, axis, lo, hi):
    s = [slice(None)] * M.dim()
    s[axis] = slice(lo, hi)
    return M[tuple(s)]


def _prim(U):
    d = U.shape[0] - 2
    v = [U[k] / U[0] for k in range(1, d + 1)]
    K = 0.5 * U[0] * sum(w * w for w in v)
    return torch.stack([U[0], *v, (GAMMA - 1) * (U[d + 1] - K)])


def _cons(W):
    d = W.shape[0] - 2
    K = 0.5 * W[0] * sum(W[k] * W[k] for k in range(1, d + 1))
    return torch.stack([W[0], *(W[0] * W[k] for k in range(1, d + 1)), W[d + 1] / (GAMMA - 1) + K])


def _flux(W, U, i):
    d = W.shape[0] - 2
    un = W[i + 1]
    F = [U[0] * un] + [U[k] * un for k in range(1, d + 1)] + [(U[d + 1] + W[d + 1]) * un]
    F[0] = W[0] * un
    F[i + 1] = F[i + 1] + W[d + 1]
    return torch.stack(F)


def _sound(W):
    c2 = GAMMA * W[-1] / W[0]
    return torch.sqrt(torch.where(c2 > MIN_C2, c2, torch.full_like(c2, MIN_C2)))


def _riemann(solver, WL, WR, UL, UR, i):
    d = WL.shape[0] - 2
    vL, vR, PL, PR = WL[i + 1], WR[i + 1], WL[d + 1], WR[d + 1]
    # selections, not maxima: at a tie the gradient goes to the selected side
    cL, cR = _sound(WL) + vL.abs(), _sound(WR) + vR.abs()
    c = torch.where(cL > cR, cL, cR)
    if solver == "llf":
        return 0.5 * (_flux(WR, UR, i) + _flux(WL, UL, i)) - 0.5 * c * (UR - UL)
    sL, sR = torch.where(vL < vR, vL, vR) - c, torch.where(vL > vR, vL, vR) + c
    rL, rR = WL[0] * (vL - sL), WR[0] * (sR - vR)
    vs = (rR * vR + rL * vL + (PL - PR)) / (rR + rL)
    phi = 1.0
    if solver == "lhllc":
        mach = torch.clamp(torch.maximum(vL.abs(), vR.abs()) / c, max=1.0)
        phi = mach * (2.0 - mach)
    Ps = (rR * PL + rL * PR + phi * rL * rR * (vL - vR)) / (rR + rL)

    def star(s, W, U, v, P):
        gap = torch.where(s == vs, torch.ones_like(s), s - vs)
        return W[0] * (s - v) / gap, ((s - v) * U[d + 1] - P * v + Ps * vs) / gap

    (aL, eL), (aR, eR) = star(sL, WL, UL, vL, PL), star(sR, WR, UR, vR, PR)

    def pick(l, ls, rs, r):
        return torch.where(sL > 0, l, torch.where(vs > 0, ls, torch.where(sR > 0, rs, r)))

    r, v = pick(WL[0], aL, aR, WR[0]), pick(vL, vs, vs, vR)
    P, e = pick(PL, Ps, Ps, PR), pick(UL[d + 1], eL, eR, UR[d + 1])
    F = [r * v] + [r * v * torch.where(vs > 0, WL[k], WR[k]) for k in range(1, d + 1)] + [v * (e + P)]
    F[i + 1] = r * v * v + P
    return torch.stack(F)


class _Plain:
    """The scheme on whole arrays; solution arrays (V, T, cells z..x, points z..x), subcell
    arrays (V, Z, Y, X)."""

    def __init__(self, case, cells, U):
        self.case, self.cells, self.d, self.p = case, cells, len(cells), case["p"]
        self.ops = _operators(self.p)
        box = PROBLEMS[case["problem"]]["box"]
        self.bc = PROBLEMS[case["problem"]]["bc"]
        self.h = [box / n for n in cells]
        self.U = U
        self.Ucv = None
        self.faces, self.centers = [], []
        for i in range(self.d):
            f = self.h[i] * np.hstack((np.repeat(np.arange(cells[i]), self.p + 1)
                                       + np.tile(self.ops["fp"][:-1], cells[i]), cells[i]))
            f = np.hstack((-f[1:3][::-1], f, f[-1] + f[1:3]))
            self.faces.append(f)
            self.centers.append(0.5 * (f[1:] + f[:-1]))

    # -- predictor ------------------------------------------------------
    def neighbours(self, M, i):
        """Left and right states at the element interfaces along i of a flux-point array."""
        lo, hi = M.select(-1 - i, 0), M.select(-1 - i, self.p + 1)
        ax = -self.d - i
        first, last = _cut(lo, ax, 0, 1), _cut(hi, ax, -1, None)
        if self.bc == "periodic":
            before, after = last, first
        else:
            before, after = first, last
            if self.bc == "reflective":
                sign = torch.ones(M.shape[0], dtype=torch.float64, device=M.device)
                sign[i + 1] = -1.0
                sign = sign.reshape((-1,) + (1,) * (first.dim() - 1))
                before, after = before * sign, after * sign
        return torch.cat([before, hi], ax), torch.cat([lo, after], ax)

    def replace_edges(self, M, X, i):
        ax = -self.d - i
        return torch.cat([_cut(X, ax, None, -1).unsqueeze(-1 - i), _cut(M, -1 - i, 1, -1),
                          _cut(X, ax, 1, None).unsqueeze(-1 - i)], -1 - i)

    def fluxes(self, Ua):
        F, M = [], []
        for i in range(self.d):
            Mi = _along(self.ops["interp"], Ua, -1 - i)
            L, R = self.neighbours(Mi, i)
            X = _riemann(self.case["solver"], _prim(L), _prim(R), L, R, i)
            F.append(self.replace_edges(_flux(_prim(Mi), Mi, i), X, i))
            M.append(Mi)
        if not self.case["viscous"]:
            return F
        Wf, dW = [], []
        for i in range(self.d):
            W = _prim(M[i])
            W = self.replace_edges(W, self.neighbours(W, i)[0], i)
            Wf.append(W)
            dW.append(_along(self.ops["deriv"], W, -1 - i) / self.h[i])
        out = []
        for i in range(self.d):
            g = []
            for e in range(self.d):
                G = _along(self.ops["interp"], dW[e], -1 - i)
                g.append(self.replace_edges(G, self.neighbours(G, i)[1], i))
            tau = [torch.zeros_like(Wf[i][0])] * (self.d + 2)
            tau[i + 1] = 2 * g[i][i + 1] - BETA * sum(g[e][e + 1] for e in range(self.d))
            # the energy part takes the normal stress before the other directions' divergence
            E = Wf[i][i + 1] * (2 - BETA) * g[i][i + 1]
            for k in range(self.d):
                if k != i:
                    tau[k + 1] = g[i][k + 1] + g[k][i + 1]
                    E = E + Wf[i][k + 1] * tau[k + 1]
            tau[self.d + 1] = E
            out.append(F[i] - torch.stack(tau) * Wf[i][0] * NU)
        return out

    def dudt(self, F, Ua):
        r = sum(_along(self.ops["deriv"], F[i], -1 - i) / self.h[i] for i in range(self.d))
        return self.gravity(r, Ua)

    def gravity(self, r, U):
        if self.case["problem"] != "column":
            return r
        r = list(r)
        r[self.d] = r[self.d] + U[0] * GRAVITY
        r[self.d + 1] = r[self.d + 1] + U[self.d] * GRAVITY
        return torch.stack(r)

    # -- one step -------------------------------------------------------
    def cfl(self):
        W = _prim(self.Ucv).detach()
        c = float((self.d * _sound(W) + W[1:self.d + 1].abs().sum(0)).max())
        h = min(self.h) / (self.p + 1)
        return CFL * (min(h / c, h * h / NU / 4) if self.case["viscous"] else h / c)

    def step(self):
        dt = self.cfl()
        Ua = self.U.unsqueeze(1).expand((self.U.shape[0], self.p + 1) + self.U.shape[1:])
        for _ in range(self.p):
            Ua = self.U.unsqueeze(1) - dt * _along(self.ops["picard"], self.dudt(self.fluxes(Ua), Ua), 1)
        F = self.fluxes(Ua)
        if self.case["update"] == "SD":
            w = _t(self.ops["weights"])
            self.U = self.U - dt * torch.tensordot(self.dudt(F, Ua), w, dims=([1], [0]))
        else:
            self.subcells(F, dt)

    def to_fv(self, M):
        order = [0]
        for i in range(self.d):
            order += [1 + i, 1 + self.d + i]
        M = M.permute(order)
        return M.reshape([M.shape[0]] + [M.shape[1 + 2 * i] * M.shape[2 + 2 * i] for i in range(self.d)])

    def to_sd(self, M):
        shape = [M.shape[0]]
        for n in self.cells[::-1]:
            shape += [n, self.p + 1]
        order = [0] + [1 + 2 * i for i in range(self.d)] + [2 + 2 * i for i in range(self.d)]
        return M.reshape(shape).permute(order)

    def ghosts(self, M, stored=None, keep=None):
        """Two ghost layers per side, direction by direction.  ``keep`` collects the layers,
        ``stored`` gives those of a side that is not refreshed."""
        for i in range(self.d):
            ax = self.d - i
            if self.bc == "periodic":
                lo, hi = _cut(M, ax, -2, None), _cut(M, ax, 0, 2)
            elif stored is not None:
                lo, hi = stored[i]
            else:
                lo, hi = _cut(M, ax, 0, 2), _cut(M, ax, -2, None)
                if self.bc == "reflective":
                    sign = torch.ones(M.shape[0], dtype=torch.float64, device=M.device)
                    sign[i + 1] = -1.0
                    sign = sign.reshape((-1,) + (1,) * self.d)
                    lo, hi = lo * sign, hi * sign
            if keep is not None:
                keep.append((lo[:1], hi[:1]))
            M = torch.cat([lo, M, hi], ax)
        return M

    def line(self, a, i):
        shape = [1] * (self.d + 1)
        shape[self.d - i] = -1
        return _t(a).reshape(shape)

    def divergence(self, U, F, dt):
        r = 0.0
        for i in range(self.d):
            ax = self.d - i
            r = r + (_cut(F[i], ax, 1, None) - _cut(F[i], ax, None, -1)) / self.line(np.diff(self.faces[i])[2:-2], i)
        return U - dt * self.gravity(r, U)

    def subcells(self, F, dt):
        d, p = self.d, self.p
        U = self.to_fv(_means(self.ops, self.U))
        high = []
        for i in range(d):
            G = F[i]
            for k in range(d):
                if k != i:
                    G = _along(self.ops["means"], G, -1 - k)
            nodes = []
            for t in range(p + 1):
                Gt = G[:, t]
                body = self.to_fv(_cut(Gt, -1 - i, 0, p + 1))
                edge = self.to_fv(_cut(_cut(Gt, -1 - i, p + 1, p + 2), -1 - d - i, -1, None))
                nodes.append(torch.cat([body, edge], d - i))
            high.append(nodes)
        for t in range(p + 1):
            dti = dt * float(self.ops["weights"][t])
            H = [high[i][t] for i in range(d)]
            W, W_new = _prim(U), _prim(self.divergence(U, H, dti))
            share = self.affected(W.detach(), W_new.detach())
            L = self.fallback(W, dti)
            U = self.divergence(U, [share[i] * L[i] + (1.0 - share[i]) * H[i] for i in range(d)], dti)
        U = self.to_sd(U)
        self.Ucv = U
        for i in range(d):
            U = _along(self.ops["points"], U, -1 - i)
        self.U = U

    # -- limiting ---------------------------------------------------------
    def affected(self, W, W_new):
        """The blended weight of the fallback flux on every face of each direction."""
        d = self.d
        kept = []
        M = self.ghosts(W, keep=kept)
        hi, lo = W, W
        for i in range(d):
            ax = d - i
            line = M
            for k in range(d):
                if k != i:
                    line = _cut(line, d - k, 2, -2)
            for a, b in ((1, -3), (3, -1)):
                side = _cut(line, ax, a, b)
                hi, lo = torch.maximum(hi, side), torch.minimum(lo, side)
        lo, hi = lo - lo.abs() * TOL, hi + hi.abs() * TOL
        bad = ~((W_new >= lo) & (W_new <= hi))
        if self.p > 1 and bool(bad.any()):
            kept = []
            N = self.ghosts(W_new, keep=kept)
            alpha = torch.ones_like(W_new)
            for i in range(d):
                line = N
                for k in range(d):
                    if k != i:
                        line = _cut(line, d - k, 2, -2)
                alpha = torch.minimum(alpha, self.smooth(line, i))
            bad = bad & (alpha < 1)
        bad = bad[0] | bad[d + 1] | ~(W_new[0] >= MIN_RHO) | ~(W_new[0] <= MAX_RHO) | ~(W_new[d + 1] >= MIN_P)
        theta = self.blend(self.ghosts(bad.double()[None], stored=kept)[0])
        out = []
        for i in range(d):
            line = theta
            for k in range(d):
                if k != i:
                    line = _cut(line, d - 1 - k, 2, -2)
            ax = d - 1 - i
            out.append(torch.maximum(_cut(line, ax, 1, -2), _cut(line, ax, 2, -1))[None])
        return out

    def smooth(self, N, i):
        """Smooth-extrema indicator along direction i (1 where the profile is smooth)."""
        ax = self.d - i
        c, h = self.centers[i], np.diff(self.faces[i])

        def slope(A, x):
            return (_cut(A, ax, 2, None) - _cut(A, ax, None, -2)) / self.line(x[2:] - x[:-2], i)

        du = slope(N, c)
        dv = 0.5 * self.line(h[2:-2], i) * slope(du, c[1:-1])
        zero = torch.zeros_like(dv)
        back = _cut(du, ax, None, -2) - _cut(du, ax, 1, -1)
        fore = _cut(du, ax, 2, None) - _cut(du, ax, 1, -1)
        aL = -torch.where(dv < 0, torch.maximum(back, zero), torch.minimum(back, zero)) / dv
        aR = torch.where(dv > 0, torch.maximum(fore, zero), torch.minimum(fore, zero)) / dv
        one = torch.ones_like(dv)
        aL, aR = (torch.where(dv == 0, one, a) for a in (aL, aR))
        aL, aR = (torch.where(a < 1, a, one) for a in (aL, aR))
        aR = torch.minimum(aL, aR)
        first = torch.cat([torch.minimum(_cut(aR, ax, None, -1), _cut(aR, ax, 1, None)), _cut(aL, ax, -1, None)], ax)
        return torch.cat([_cut(first, ax, None, 1), torch.minimum(_cut(aR, ax, None, -1), _cut(first, ax, 1, None))], ax)

    def blend(self, t):
        """Weights around troubled subcells, the neighbour pairs of the reference scheme."""
        d, th = self.d, t.clone()
        a, b = slice(None, -1), slice(1, None)

        def at(i, s):
            r = [slice(None)] * d
            r[d - 1 - i] = s
            return tuple(r)

        for i in range(d):
            th[at(i, a)] = torch.maximum(0.75 * t[at(i, b)], th[at(i, a)])
            th[at(i, b)] = torch.maximum(0.75 * t[at(i, a)], th[at(i, b)])
        pairs = [(a, a), (a, b), (b, a), (b, b)]
        if d == 2:
            for k in range(4):
                th[pairs[k]] = torch.maximum(0.5 * t[pairs[3 - k]], th[pairs[k]])
        elif d == 3:
            for k in range(4):
                for i in range(3):
                    to, frm = [slice(None), *pairs[k]], [slice(None), *pairs[::-1][-k]]
                    to, frm = tuple(to[i:] + to[:i]), tuple(frm[i:] + frm[:i])
                    th[to] = torch.maximum(0.5 * t[frm], th[to])
            for y in (a, b):
                for x in (a, b):
                    frm = (b, b if y is a else a, b if x is a else a)
                    th[(a, y, x)] = torch.maximum(0.375 * t[frm], th[(a, y, x)])
        for i in range(d):
            th[at(i, a)] = torch.maximum(0.25 * (th[at(i, b)] > 0).double(), th[at(i, a)])
            th[at(i, b)] = torch.maximum(0.25 * (th[at(i, a)] > 0).double(), th[at(i, b)])
        return th

    def limited(self, L, R, xl, xr, xm):
        if self.case["slopes"] == "minmod":
            r = (R / torch.where(L == 0, torch.ones_like(L), L)).detach()
            mid = torch.where((r > 0) & (r < 1) & (L != 0), R, L)
            return torch.where((r <= 0) & (L != 0), torch.zeros_like(L), mid)
        c = (xl * L + xr * R) / (xl + xr)
        s = torch.minimum(torch.minimum((2 * L * xl / xm).abs(), (2 * R * xr / xm).abs()), c.abs())
        return torch.where(L * R >= 0, torch.sign(c).detach() * s, torch.zeros_like(c))

    def fallback(self, W, dt):
        """MUSCL-Hancock fluxes of every face."""
        d = self.d
        M = self.ghosts(W)
        inner = M
        for i in range(d):
            inner = _cut(inner, d - i, 1, -1)
        grads, slopes = [], []
        for i in range(d):
            ax = d - i
            line = M
            for k in range(d):
                if k != i:
                    line = _cut(line, d - k, 1, -1)
            hc, hf = np.diff(self.centers[i]), np.diff(self.faces[i])
            g = (_cut(line, ax, 1, None) - _cut(line, ax, None, -1)) / self.line(hc, i)
            g = self.limited(_cut(g, ax, None, -1), _cut(g, ax, 1, None), self.line(hc[:-1], i), self.line(hc[1:], i),
                             self.line(hf[1:-1], i))
            grads.append(g)
            slopes.append(0.5 * g * self.line(hf[1:-1], i))
        rate = [0.0] * (d + 2)
        for i in range(d):
            g, v = grads[i], inner[i + 1]
            rate[0] = rate[0] - v * g[0] - inner[0] * g[i + 1]
            rate[i + 1] = rate[i + 1] - v * g[i + 1] - g[d + 1] / inner[0]
            # the transverse terms as the reference has them, over all but the first velocity
            for k in range(2, d + 1):
                rate[k] = rate[k] - v * g[k]
        rate[d + 1] = torch.zeros_like(inner[0])
        half = inner + 0.5 * dt * torch.stack(rate)
        out = []
        for i in range(d):
            ax = d - i
            lo, hi = half + slopes[i], half - slopes[i]
            for k in range(d):
                if k != i:
                    lo, hi = _cut(lo, d - k, 1, -1), _cut(hi, d - k, 1, -1)
            WL, WR = _cut(lo, ax, None, -1), _cut(hi, ax, 1, None)
            out.append(_riemann(self.case["solver"], WL, WR, _cons(WL), _cons(WR), i))
        return out


def exact(case, seed):
    outs = []
    for cells, s in _members(case, seed):
        U = _t(_initial(case, cells, s))
        if case["api"] == "gradient":
            U.requires_grad_(True)
        with torch.set_grad_enabled(case["api"] == "gradient"):
            sim = _Plain(case, cells, U)
            sim.Ucv = _means(sim.ops, U.detach())
            for _ in range(case["steps"]):
                sim.step()
            outs.append(sim)
    if case["api"] == "ensemble":
        return [o.U for o in outs]
    end = outs[0].U
    if case["api"] == "gradient":
        g = torch.Generator(device=DEVICE).manual_seed(int(seed))
        dy = torch.randn(U.shape, dtype=torch.float64, device=DEVICE, generator=g)
        (grad,) = torch.autograd.grad(end, U, dy)
        return {"U": end.detach(), "grad": grad}
    if case["api"] == "host":
        return {"U": end, "W": _prim(_means(outs[0].ops, end))}
    return end
