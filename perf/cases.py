"""Timed workloads of the framework, through its public Python entry points.

Each case is a dict of plain values.  `prepare` builds what a user's program
holds before the call (the problem's arrays and the open session), `run` is
one call as that program makes it, and `exact` is the same computation in
plain torch at 64 bits, written from the scheme (unsplit MUSCL-Hancock or
first-order Godunov, HLLC or the exact Riemann solver), without this
package's code.

Kinds of call:

  launch    Simulation2D: reset the host arrays and call launch_simulation
            (host arrays in and out), as a program written against the C API
  session   Solver2D: rewind the device-resident session, advance, download
  batch     Batch2D: the same for an ensemble of independent grids
  adjoint   Adjoint2D: forward pass and the gradient of a scalar objective
  run_1d    run_1d: one whole 1D run

Problems (hydrofv_gb300.problems): shear layer, point blast, Rayleigh-Taylor,
smooth waves with noise, four-quadrant Riemann problems, Sod and Sedov.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import hydrofv_gb300 as H
from hydrofv_gb300 import problems as P

LIMITERS = ("minmod", "van_leer", "monotonized_central")


# ------------------------------------------------------------------ cases

def listed():
    return [
        # the smallest call a program makes: a 64^2 grid for a few steps, host arrays in and out
        {"name": "shear 64 launch", "kind": "launch", "problem": "shear", "nx": 64, "ny": 64,
         "limiter": "monotonized_central", "steps": 20},
        # an example program of the original code at its own size, with gravity and three ghost layers
        {"name": "rayleigh-taylor 122 launch", "kind": "launch", "problem": "rayleigh_taylor", "nx": 122, "ny": 122,
         "limiter": "monotonized_central", "steps": 200},
        # an ordinary mid-size run on a ragged grid, walls in x and outflow in y
        {"name": "waves 401x250 session", "kind": "session", "problem": "waves", "nx": 401, "ny": 250,
         "bc": "reflective,transmissive", "limiter": "van_leer", "steps": 200, "fp32": False},
        # a blast wave, mostly undisturbed gas, walls all round
        {"name": "blast 1024 launch", "kind": "launch", "problem": "blast", "nx": 1024, "ny": 1024,
         "limiter": "van_leer", "steps": 100},
        # the benchmark's shear layer at full size, end to end
        {"name": "shear 2048 launch", "kind": "launch", "problem": "shear", "nx": 2048, "ny": 2048,
         "limiter": "monotonized_central", "steps": 100},
        # the FP32 state form on a small ragged grid
        {"name": "waves 301x200 fp32", "kind": "session", "problem": "waves", "nx": 301, "ny": 200,
         "bc": "periodic,periodic", "limiter": "monotonized_central", "steps": 500, "fp32": True},
        # the FP32 state form at the benchmark's size
        {"name": "shear 2048 fp32", "kind": "session", "problem": "shear", "nx": 2048, "ny": 2048,
         "bc": "periodic,periodic", "limiter": "monotonized_central", "steps": 600, "fp32": True},
        # ensembles of uneven grids, each with its own time step
        {"name": "ensemble 24 fp64", "kind": "batch", "count": 24, "side_lo": 128, "side_hi": 512,
         "limiter": "minmod", "steps": 60, "fp32": False},
        {"name": "ensemble 28 fp32", "kind": "batch", "count": 28, "side_lo": 128, "side_hi": 640,
         "limiter": "minmod", "steps": 200, "fp32": True},
        # forward and backward: the gradient of a scalar with respect to the initial state
        {"name": "adjoint 192", "kind": "adjoint", "nx": 192, "limiter": "monotonized_central", "steps": 40, "every": 10},
        # the benchmark's shock tube, one whole run with the exact Riemann solver
        {"name": "sod 1000", "kind": "run_1d", "problem": "sod", "nx": 1000, "steps": -1},
        # a spherical blast with the geometry source
        {"name": "sedov spherical 508", "kind": "run_1d", "problem": "sedov", "nx": 508, "steps": 400},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges."""
    kind = rng.choice(["launch", "launch", "session", "session", "session", "batch", "adjoint", "run_1d"])
    limiter = rng.choice(LIMITERS)
    if kind == "launch":
        problem = rng.choice(["shear", "rayleigh_taylor", "blast", "waves"])
        n = _log_int(rng, 48, 1500)
        ny = n if problem in ("shear", "blast") else max(40, int(n * rng.uniform(0.5, 2.0)))
        steps = max(10, min(200, int(2e8 / (n * ny))))
        c = {"kind": kind, "problem": problem, "nx": n, "ny": ny, "limiter": limiter, "steps": steps}
        if problem == "waves":
            c["bc"] = ",".join(rng.choice(["periodic", "reflective", "transmissive"]) for _ in range(2))
            c["first_order"] = rng.random() < 0.3
        return c
    if kind == "session":
        fp32 = rng.random() < 0.5
        problem = rng.choice(["shear", "waves"])
        n = _log_int(rng, 48, 1800)
        ny = n if problem == "shear" else max(40, int(n * rng.uniform(0.5, 2.0)))
        steps = max(20, min(500, int((1.5e9 if fp32 else 2e8) / (n * ny))))
        bc = ",".join(rng.choice(["periodic", "reflective", "transmissive"]) for _ in range(2))
        return {"kind": kind, "problem": problem, "nx": n, "ny": ny, "limiter": limiter, "steps": steps, "fp32": fp32,
                "bc": "periodic,periodic" if problem == "shear" else bc}
    if kind == "batch":
        fp32 = rng.random() < 0.5
        lo = rng.randrange(64, 200)
        return {"kind": kind, "count": rng.randrange(4, 24), "side_lo": lo, "side_hi": rng.randrange(200, 500),
                "limiter": limiter, "steps": rng.randrange(20, 60) * (3 if fp32 else 1), "fp32": fp32}
    if kind == "adjoint":
        every = rng.randrange(4, 12)
        return {"kind": kind, "nx": _log_int(rng, 48, 256), "limiter": limiter, "steps": every * rng.randrange(2, 4),
                "every": every}
    problem = rng.choice(["sod", "sedov"])
    n = _log_int(rng, 100, 1000)
    return {"kind": kind, "problem": problem, "nx": n, "steps": -1 if problem == "sod" else rng.randrange(100, 400)}


# ----------------------------------------------------------------- inputs

def _scale_2d(p, rng):
    """Other inputs for another seed: small random factors on density and pressure."""
    W = p.W.copy()
    W[0] *= 1.0 + 0.05 * rng.uniform(-1.0, 1.0)
    W[3] *= 1.0 + 0.05 * rng.uniform(-1.0, 1.0)
    p.W = W
    p.U = P.primitive_to_conserved_2d(W, p.gamma, p.dx * p.dy)
    return p


def _problem_2d(case, seed):
    rng = np.random.default_rng(seed)
    kind, nx, ny, steps = case["problem"], case["nx"], case["ny"], case["steps"]
    if kind == "shear":
        p = P.shear_layer(nx, seed=int(seed), steps=steps)
    elif kind == "rayleigh_taylor":
        p = _scale_2d(P.rayleigh_taylor(nx, ny, steps=steps), rng)
    elif kind == "blast":
        p = _scale_2d(P.point_blast(nx, steps=steps), rng)
    else:
        x, y = case["bc"].split(",")
        p = P.random_problem_2d(nx, ny, int(seed), (x, x, y, y), case["limiter"], steps, smooth=True,
                                integrator="godunov_first_order_2d" if case.get("first_order") else "muscl_hancock_2d")
    p.slope_limiter = case["limiter"]
    return p


def _ensemble(case, seed):
    rng = np.random.default_rng(4)   # the grids are the case's; the states are the seed's
    sides = np.rint(np.exp(rng.uniform(math.log(case["side_lo"]), math.log(case["side_hi"]), size=case["count"])))
    rng = np.random.default_rng(seed)
    return [P.four_quadrant(int(s), rng, steps=case["steps"], limiter=case["limiter"]) for s in sides]


def _adjoint_problem(case, seed):
    return P.shear_layer(case["nx"], seed=int(seed), steps=case["steps"], limiter=case["limiter"], rho_p_noise=1e-3)


def _problem_1d(case, seed):
    rng = np.random.default_rng(seed)
    if case["problem"] == "sedov":
        p = P.sedov_1d(case["nx"] + 4, coord_sys="spherical_1d", steps=case["steps"])
        p.U = p.U * (1.0 + 0.05 * rng.uniform(-1.0, 1.0))   # a heavier or lighter gas at the same speeds
        p.W = p.W.copy()
        f = p.U[0, 2] / (p.W[0, 2] * P.geometry_1d(p.x_min, p.x_max, p.nx, p.g, p.coord_sys)[1][2])
        p.W[0] *= f
        p.W[2] *= f
        return p
    p = P.sod_1d(case["nx"])
    W = p.W.copy()
    left = W[0] > 0.5
    W[0] = np.where(left, 1.0 + 0.1 * rng.uniform(), 0.125 + 0.02 * rng.uniform())
    W[2] = np.where(left, 1.0 + 0.1 * rng.uniform(), 0.1 + 0.02 * rng.uniform())
    p.W, p.U = W, P.primitive_to_conserved_1d(W, p.gamma, 1.0 / (p.nx + 2 * p.g))
    return p


class _State:
    """A problem and the open session on it, closed with the last reference
    (a launch's System goes with the last array that shows it)."""

    def __init__(self, kind, problem, handle=None):
        self.kind, self.problem, self.handle = kind, problem, handle

    def __del__(self):
        if self.handle is not None and self.kind != "launch":
            self.handle.close()


def _system_arrays(system, names):
    """The System's own host arrays, where a launch leaves its result; each keeps the System alive."""
    out = []
    for name in names:
        buf = (ctypes.c_double * system.n).from_address(ctypes.addressof(getattr(system.s, name).contents))
        buf.system = system
        out.append(np.frombuffer(buf, dtype=np.float64).reshape(system.shape))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "run_1d":
        return _State(kind, _problem_1d(case, seed))
    opts = H.default_options(precision=1 if case.get("fp32") else 0)
    if kind == "batch":
        ps = _ensemble(case, seed)
        st = _State(kind, ps, H.Batch2D(ps, options=opts))
        st.steps, st.fp32 = case["steps"], case["fp32"]
        return st
    if kind == "adjoint":
        p = _adjoint_problem(case, seed)
        return _State(kind, p, H.Adjoint2D(p, case["steps"], case["every"], options=opts))
    p = _problem_2d(case, seed)
    bounds = (p.x_min, p.x_max, p.y_min, p.y_max)
    if kind == "launch":
        h = H.Simulation2D(p.nx, p.ny, p.g, bounds, p.gamma, p.W, p.U, bc=p.bc, integrator=p.integrator,
                           slope_limiter=p.slope_limiter, cfl=p.cfl, tf=p.tf, max_steps=p.max_steps, options=opts,
                           gravity=p.gravity)
        st = _State(kind, p, h)
        st.W, st.U = _system_arrays(h.h, H.W2), _system_arrays(h.h, H.U2)
        return st
    st = _State(kind, p, H.Solver2D(p.nx, p.ny, p.g, bounds, p.gamma, p.W, p.U, bc=p.bc, slope_limiter=p.slope_limiter,
                                    cfl=p.cfl, options=opts, gravity=p.gravity))
    st.fp32 = case["fp32"]
    return st


def run(state):
    kind, p, h = state.kind, state.problem, state.handle
    if kind == "launch":
        h.load(p.W, p.U)
        code, msg, st, _ = h.launch()
        if code != 0:
            raise RuntimeError(msg)
        return {"W": state.W, "U": state.U, "steps": int(st.num_steps), "t": float(st.t), "dt": float(st.dt)}
    if kind == "session":
        h.restart()
        st, _ = h.advance(p.max_steps)
        W, U = h.download()
        if state.fp32:   # the FP32 form's state: float32 values, kept as such
            W, U = W.astype(np.float32), U.astype(np.float32)
        return {"W": W, "U": U, "steps": int(st.num_steps), "t": float(st.t), "dt": float(st.dt)}
    if kind == "batch":
        h.restart()
        sts, _ = h.advance(state.steps)
        out = h.download()
        if state.fp32:
            out = [(W.astype(np.float32), U.astype(np.float32)) for W, U in out]
        return {"state": out, "steps": np.array([s[0] for s in sts]), "t": np.array([s[1] for s in sts]),
                "dt": np.array([s[2] for s in sts])}
    if kind == "adjoint":
        W = h.forward()
        J, seed = P.right_half_density_squared(p, W)
        return {"W": W, "J": J, "grad": h.backward(seed)}
    r = H.run_1d(p.nx, p.g, (p.x_min, p.x_max), p.gamma, p.W, p.U, bc=p.bc, integrator=p.integrator,
                 riemann_solver=p.riemann_solver, slope_limiter=p.slope_limiter, cfl=p.cfl, tf=p.tf,
                 max_steps=p.max_steps, coord_sys=p.coord_sys)
    if r.code != 0:
        raise RuntimeError(r.message)
    return {"W": r.W, "U": r.U, "steps": r.num_steps, "t": r.t, "dt": r.dt}


def work(case):
    """Every step reads and writes the conserved state once; about 400
    additions and multiplications per cell-update in 2D (two
    reconstructions, two HLLC faces, update), 250 in 1D with HLLC and 600
    with the exact solver, 1500 for forward, recomputation and reverse."""
    kind = case["kind"]
    if kind == "batch":
        rng = np.random.default_rng(4)
        sides = np.rint(np.exp(rng.uniform(math.log(case["side_lo"]), math.log(case["side_hi"]), size=case["count"])))
        cells, steps = float((sides * sides).sum()), case["steps"]
    elif kind == "run_1d":
        cells = case["nx"]
        # wave speed of the Sod states about 2.2, CFL 0.9, tf = 0.2
        steps = case["steps"] if case["steps"] > 0 else 0.2 * 2.2 * cells / 0.9
        return {"bytes": 2 * 3 * 8.0 * cells * steps, "flops": (600.0 if case["problem"] == "sod" else 250.0) * cells * steps}
    elif kind == "adjoint":
        cells, steps = case["nx"] ** 2, case["steps"]
        return {"bytes": 3 * 64.0 * cells * steps, "flops": 1500.0 * cells * steps}
    else:
        cells, steps = case["nx"] * case["ny"], case["steps"]
    return {"bytes": (32.0 if case.get("fp32") else 64.0) * cells * steps, "flops": 400.0 * cells * steps}


# ------------------------------------------------------ the scheme, 64 bits

_TOL = 1e-6                  # IntegratorParam's default tolerance
_SHRINK, _SHRINK_STEPS = 0.2, 10


def _slope(lim, a, b):
    zero = torch.zeros_like(a)
    same = a * b > 0
    if lim == "minmod":
        s = torch.where(a.abs() < b.abs(), a, b)
    elif lim == "van_leer":
        s = 2.0 * a * b / torch.where(same, a + b + 1e-10, torch.ones_like(a))
    else:
        s = torch.sign(a) * torch.minimum(0.5 * (a + b).abs(), 2.0 * torch.minimum(a.abs(), b.abs()))
    return torch.where(same, s, zero)


def _sound(g, rho, p):
    return torch.where(rho > 0, torch.sqrt(g * p / rho), torch.zeros_like(rho))


def _vacuum_state(g, L, R, aL, aR, side):
    """The state at x/t = 0 of a problem with vacuum: `side` picks the right-vacuum sampler (fan of L) or the left one."""
    rho, u, v, p = L if side == "right" else R
    a, s = (aL, 1.0) if side == "right" else (aR, -1.0)
    base = 2.0 / (g + 1.0) + s * u * (g - 1.0) / ((g + 1.0) * a)
    k = base ** (2.0 / (g - 1.0))
    fan = [rho * k, (s * a + 0.5 * (g - 1.0) * u) * 2.0 / (g + 1.0), v, p * base ** (2.0 * g / (g - 1.0))]
    inside = s * (u + s * 2.0 * a / (g - 1.0)) > 0
    still = s * (u - s * a) >= 0
    z = torch.zeros_like(rho)
    return [torch.where(still, w, torch.where(inside, f, z)) for w, f in zip((rho, u, v, p), fan)]


def _guess(g, L, R, aL, aR):
    rL, uL, _, pL = L
    rR, uR, _, pR = R
    lo, hi = torch.minimum(pL, pR), torch.maximum(pL, pR)
    ppv = 0.5 * (pL + pR) - 0.125 * (uR - uL) * (rL + rR) * (aL + aR)
    z = 0.5 * (g - 1.0) / g
    trrs = ((aL + aR - 0.5 * (g - 1.0) * (uR - uL)) / (aL / pL ** z + aR / pR ** z)) ** (1.0 / z)
    k = (g - 1.0) / (g + 1.0)
    gL = torch.sqrt(2.0 / ((g + 1.0) * rL) / (ppv + k * pL))
    gR = torch.sqrt(2.0 / ((g + 1.0) * rR) / (ppv + k * pR))
    tsrs = (gL * pL + gR * pR - (uR - uL)) / (gL + gR)
    mild = (hi / lo <= 2.0) & (lo <= ppv) & (ppv <= hi)
    return torch.where(mild, ppv, torch.where(ppv < lo, trrs, tsrs)).clamp(min=_TOL)


def _hllc(g, L, R):
    """Flux (mass, normal, tangential momentum, energy) of states (rho, u_n, u_t, p)."""
    rL, uL, vL, pL = L
    rR, uR, vR, pR = R
    aL, aR = _sound(g, rL, pL), _sound(g, rR, pR)
    vac = (rL <= 0) | (rR <= 0) | (2.0 * (aL + aR) / (g + 1.0) <= uR - uL)
    ps = _guess(g, L, R, aL, aR)

    def q(p):
        return torch.where(ps <= p, torch.ones_like(p), torch.sqrt((1.0 + (0.5 + 0.5 / g) * (ps / p - 1.0)).clamp(min=0.0)))
    SL, SR = uL - aL * q(pL), uR + aR * q(pR)
    Ss = (pR - pL + rL * uL * (SL - uL) - rR * uR * (SR - uR)) / (rL * (SL - uL) - rR * (SR - uR))
    left = (SL >= 0) | (Ss >= 0)
    star = (SL < 0) & (SR > 0)
    rho, u, v, p = (torch.where(left, x, y) for x, y in zip(L, R))
    S = torch.where(left, SL, SR)
    E = rho * (0.5 * (u * u + v * v)) + p / (g - 1.0)
    rs = rho * (S - u) / (S - Ss)
    es = rs * (E / rho + (Ss - u) * (Ss + p / (rho * (S - u))))
    F = [rho * u, rho * u * u + p, rho * u * v, u * (E + p)]
    D = [rs - rho, rs * Ss - rho * u, rs * v - rho * v, es - E]
    F = [torch.where(star, f + S * d, f) for f, d in zip(F, D)]
    if bool(vac.any()):
        SvL, SvR = 2.0 * aL / (g - 1.0), 2.0 * aR / (g - 1.0)
        r, l = _vacuum_state(g, L, R, aL, aR, "right"), _vacuum_state(g, L, R, aL, aR, "left")
        pick_r, pick_l = (rL <= 0) | ((rR > 0) & (SvL >= 0)), (rR <= 0) | (SvR <= 0)
        both = (rL <= 0) & (rR <= 0)
        s = [torch.where(both, torch.zeros_like(x), torch.where(pick_r, x, torch.where(pick_l, y, torch.zeros_like(x))))
             for x, y in zip(r, l)]
        e = s[0] * 0.5 * (s[1] ** 2 + s[2] ** 2) + s[3] / (g - 1.0)
        V = [s[0] * s[1], s[0] * s[1] ** 2 + s[3], s[0] * s[1] * s[2], s[1] * (e + s[3])]
        F = [torch.where(vac, x, y) for x, y in zip(V, F)]
    return F


def _predict(g, lim, W, dtA, axis):
    """Half-step states at the low and high face of every cell but the first and last along `axis` (0: y, 1: x)."""
    n = W[0].shape[axis]
    lo_, mid_, hi_ = (lambda f, k=k: f.narrow(axis, k, n - 2) for k in (0, 1, 2))
    rho, u, v, p = (mid_(f) for f in W)
    d = [_slope(lim, mid_(f) - lo_(f), hi_(f) - mid_(f)) for f in W]
    un, dn = (u, d[1]) if axis == 1 else (v, d[2])
    a2 = g * p / rho
    both = []
    for s in (-1.0, 1.0):
        k = 1.0 - s * dtA * un
        # the density row takes the slope of the x velocity in both sweeps
        r_ = rho + s * 0.5 * (k * d[0] - s * dtA * rho * d[1])
        p_ = p + s * 0.5 * (k * d[3] - s * dtA * rho * a2 * dn)
        n_ = un + s * 0.5 * (k * dn - s * dtA / rho * d[3])
        t, dt_ = (v, d[2]) if axis == 1 else (u, d[1])
        both.append([r_, n_, t + s * 0.5 * k * dt_, p_])
    return both


def _bc(W, G, nx, ny, bc):
    for axis, n, names, normal in ((1, nx, bc[:2], 1), (0, ny, bc[2:], 2)):
        other = slice(G, G + (ny if axis == 1 else nx))

        def at(f, i):
            return (f, (other, i)) if axis == 1 else (f, (i, other))
        for side in (0, 1):
            for k in range(G):
                dst = G - 1 - k if side == 0 else G + n + k
                if names[side] == "periodic":
                    src = G + n - 1 - k if side == 0 else G + k
                else:
                    src = G + k if side == 0 else G + n - 1 - k
                for q, f in enumerate(W):
                    x = f[at(f, src)[1]]
                    f[at(f, dst)[1]] = -x if names[side] == "reflective" and q == normal else x


def _solve_2d(p, steps):
    """(W, U, t, dt) after `steps` steps from the padded arrays of a Problem2D-like p, in float64."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g, G, nx, ny = p.gamma, p.g, p.nx, p.ny
    dx, dy = (p.x_max - p.x_min) / (nx + 2 * G), (p.y_max - p.y_min) / (ny + 2 * G)
    vol = dx * dy
    W = [torch.from_numpy(np.ascontiguousarray(f)).to(dev, torch.float64) for f in p.W]
    U = [torch.from_numpy(np.ascontiguousarray(f)).to(dev, torch.float64) for f in p.U]
    I, J = slice(G, G + ny), slice(G, G + nx)
    first_order = p.integrator == "godunov_first_order_2d"
    t = torch.zeros((), dtype=torch.float64, device=dev)
    dt = t
    for n in range(steps):
        rho, u, v, pr = (f[I, J] for f in W)
        a = torch.sqrt(g * pr / rho)
        cfl = p.cfl * (_SHRINK if n < _SHRINK_STEPS else 1.0)
        dt = cfl / ((a + u.abs()).max() / dx + (a + v.abs()).max() / dy)
        xs = [f[I, G - 2:G + nx + 2] for f in W]
        ys = [f[G - 2:G + ny + 2, J] for f in W]
        if first_order:
            xlo = xhi = [f[:, 1:-1] for f in xs]
            ylo = yhi = [f[1:-1] for f in (ys[0], ys[2], ys[1], ys[3])]
        else:
            xlo, xhi = _predict(g, p.slope_limiter, xs, dt * dy / vol, 1)
            ylo, yhi = _predict(g, p.slope_limiter, ys, dt * dx / vol, 0)
        F = _hllc(g, [f[:, :-1] for f in xhi], [f[:, 1:] for f in xlo])
        K = _hllc(g, [f[:-1] for f in yhi], [f[1:] for f in ylo])
        K = [K[0], K[2], K[1], K[3]]
        for q in range(4):
            fx, fy = F[q] * dt * dy, K[q] * dt * dx
            U[q][I, G:G + nx + 1] += fx
            U[q][I, G - 1:G + nx] -= fx
            U[q][G:G + ny + 1, J] += fy
            U[q][G - 1:G + ny, J] -= fy
        if p.gravity:
            # RK4 on the energy of the uniform acceleration (interior cells)
            m, my = U[0][I, J], U[2][I, J]
            k = -dt * p.gravity
            U[3][I, J] += k * (my + 0.5 * k * m)
            U[2][I, J] += k * m
        w1, w2 = U[1] / U[0], U[2] / U[0]
        W = [U[0] / vol, w1, w2, (g - 1.0) * (U[3] - 0.5 * U[0] * (w1 * w1 + w2 * w2)) / vol]
        _bc(W, G, nx, ny, p.bc)
        t = t + dt
    return W, U, float(t), float(dt)


def _star(g, rho_L, u_L, p_L, a_L, rho_R, u_R, p_R, a_R):
    """p* by Newton's method from the guess, until its relative change is below the tolerance."""
    z = torch.zeros_like(rho_L)
    p = _guess(g, (rho_L, u_L, z, p_L), (rho_R, u_R, z, p_R), a_L, a_R)

    def f(rho, pk, a, ps):
        A, B = 2.0 / ((g + 1.0) * rho), pk * (g - 1.0) / (g + 1.0)
        return torch.where(ps > pk, (ps - pk) * torch.sqrt(A / (ps + B)),
                           2.0 * a / (g - 1.0) * ((ps / pk) ** ((g - 1.0) / (2.0 * g)) - 1.0))

    def df(rho, pk, a, ps):
        A, B = 2.0 / ((g + 1.0) * rho), pk * (g - 1.0) / (g + 1.0)
        return torch.where(ps > pk, (1.0 - 0.5 * (ps - pk) / (B - ps)) * torch.sqrt(A / (B + ps)),
                           (ps / pk) ** (-0.5 * (g + 1.0) / g) / (pk * a))
    done = torch.zeros_like(rho_L, dtype=torch.bool)
    for _ in range(100):
        r = f(rho_L, p_L, a_L, p) + f(rho_R, p_R, a_R, p) + (u_R - u_L)
        q = p - r / (df(rho_L, p_L, a_L, p) + df(rho_R, p_R, a_R, p))
        near = 2.0 * (q - p).abs() / (q + p) < _TOL
        p = torch.where(done, p, q)
        done = done | near
        if bool(done.all()):
            break
    us = 0.5 * (u_L + u_R) + 0.5 * (f(rho_R, p_R, a_R, p) - f(rho_L, p_L, a_L, p))
    return p, us


def _exact_flux(g, L, R):
    """Godunov flux of the exact Riemann solution at x/t = 0 (no vacuum)."""
    a_L, a_R = torch.sqrt(g * L[2] / L[0]), torch.sqrt(g * R[2] / R[0])
    ps, us = _star(g, *L, a_L, *R, a_R)
    left = us > 0
    rho, u, p, a = (torch.where(left, x, y) for x, y in zip((*L, a_L), (*R, a_R)))
    s = torch.where(left, torch.ones_like(us), -torch.ones_like(us))   # mirror the right side onto the left
    u, um = s * u, s * us
    r, k = ps / p, (g - 1.0) / (g + 1.0)
    shock = ps > p
    speed = u - a * torch.sqrt((g + 1.0) / (2.0 * g) * r + (g - 1.0) / (2.0 * g))
    head, tail = u - a, um - a * r ** ((g - 1.0) / (2.0 * g))
    c = 2.0 / (g + 1.0) + u * (g - 1.0) / (a * (g + 1.0))
    fan = [rho * c ** (2.0 / (g - 1.0)), 2.0 / (g + 1.0) * (a + 0.5 * u * (g - 1.0)), p * c ** (2.0 * g / (g - 1.0))]
    star = [torch.where(shock, rho * (r + k) / (k * r + 1.0), rho * r ** (1.0 / g)), um, ps]
    undisturbed = torch.where(shock, speed > 0, head > 0)
    in_fan = ~shock & (head <= 0) & (tail > 0)
    o = [torch.where(undisturbed, w, torch.where(in_fan, f, x)) for w, f, x in zip((rho, u, p), fan, star)]
    o[1] = s * o[1]
    return [o[0] * o[1], o[0] * o[1] ** 2 + o[2], (o[2] * g / (g - 1.0) + 0.5 * o[0] * o[1] ** 2) * o[1]]


def _solve_1d(p):
    """(W, U, steps, t, dt) of a 1D run to tf or max_steps, in float64 on the CPU."""
    g, G, n = p.gamma, p.g, p.nx
    tot = n + 2 * G
    dx = (p.x_max - p.x_min) / tot
    r = p.x_min + np.arange(tot + 1) * dx
    alpha = {"cartesian_1d": 0.0, "cylindrical_1d": 1.0, "spherical_1d": 2.0}[p.coord_sys]
    area, vol = np.ones(tot + 1), np.full(tot, dx)
    if alpha == 1.0:
        area, vol = 2 * math.pi * r, math.pi * (r[1:] ** 2 - r[:-1] ** 2)
    if alpha == 2.0:
        area, vol = 4 * math.pi * r ** 2, 4.0 / 3.0 * math.pi * (r[1:] ** 3 - r[:-1] ** 3)
    area, vol = torch.from_numpy(area)[:tot], torch.from_numpy(vol)
    mid = torch.from_numpy(p.x_min + (np.arange(tot) + 0.5) * dx)
    W = [torch.from_numpy(f.copy()) for f in p.W]
    U = [torch.from_numpy(f.copy()) for f in p.U]
    I = slice(G, G + n)

    def primitive():
        u = U[1] / U[0]
        w = [U[0] / vol, u, (g - 1.0) * (U[2] - 0.5 * U[0] * u * u) / vol]
        for side in (0, 1):
            for k in range(G):
                dst, src = (G - 1 - k, G + k) if side == 0 else (G + n + k, G + n - 1 - k)
                for q in range(3):
                    w[q][dst] = -w[q][src] if q == 1 and p.bc[side] == "reflective" else w[q][src]
        return w

    def rates(pf, m, q, e):
        pr = (g - 1.0) * (e - 0.5 * q * q / m)
        return pf * q, pf * q * q / m, pf * q * (e + pr) / m
    t, dt, steps = 0.0, 0.0, 0
    while t < p.tf and (p.max_steps < 0 or steps < p.max_steps):
        rho, u, pr = (f[I] for f in W)
        cfl = p.cfl * (_SHRINK if steps < _SHRINK_STEPS else 1.0)
        dt = cfl * dx / float((torch.sqrt(g * pr / rho) + u.abs()).max())
        if t + dt > p.tf:
            dt = p.tf - t
        if p.integrator == "muscl_hancock_1d":
            z = torch.zeros(1, tot, dtype=torch.float64)
            k = slice(G - 2, G + n + 2)
            X = [f[None, k] for f in (W[0], W[1], z[0], W[2])]
            dtA = (dt * area / vol)[None, G - 1:G + n + 1]
            lo, hi = _predict(g, p.slope_limiter, X, dtA, 1)
            F = _hllc(g, [f[:, :-1] for f in hi], [f[:, 1:] for f in lo])
            F = [F[0][0], F[1][0], F[3][0]]
        else:
            F = _exact_flux(g, [f[G - 1:G + n] for f in W], [f[G:G + n + 1] for f in W])
        for q in range(3):
            U[q][G:G + n + 1] += F[q] * dt * area[G:G + n + 1]
            U[q][G - 1:G + n] -= F[q] * dt * area[G - 1:G + n]
        W = primitive()
        if alpha:
            # RK4 of the geometry source on the interior totals; the first stage takes the density just converted
            v, pf = vol[I], -alpha * vol[I] / mid[I]
            y0 = [f[I].clone() for f in U]
            y, ks = y0, []
            for c in (0.5, 0.5, 1.0, None):
                ks.append(rates(pf, *[f / v for f in y]))
                if c is not None:
                    y = [a + c * dt * b for a, b in zip(y0, ks[-1])]
            for q in range(3):
                U[q][I] = y0[q] + dt * (ks[0][q] + 2.0 * ks[1][q] + 2.0 * ks[2][q] + ks[3][q]) / 6.0
            W = primitive()
        t, steps = t + dt, steps + 1
    return torch.stack(W).numpy(), torch.stack(U).numpy(), steps, t, dt


def exact(case, seed):
    """What run returns, from the scheme in plain torch at 64 bits; None where that would take too long."""
    kind = case["kind"]
    if work(case)["flops"] / 400.0 > 5e8:
        return None
    if kind == "run_1d":
        W, U, steps, t, dt = _solve_1d(_problem_1d(case, seed))
        return {"W": W, "U": U, "steps": steps, "t": t, "dt": dt}
    if kind == "batch":
        if case["count"] * case["steps"] > 3000:
            return None
        got = [_solve_2d(p, case["steps"]) for p in _ensemble(case, seed)]
        return {"state": [(torch.stack(W), torch.stack(U)) for W, U, _, _ in got],
                "steps": np.full(case["count"], case["steps"]), "t": np.array([x[2] for x in got]),
                "dt": np.array([x[3] for x in got])}
    if kind == "adjoint":
        p = _adjoint_problem(case, seed)
        W = torch.stack(_solve_2d(p, case["steps"])[0]).cpu().numpy()
        out = np.zeros_like(W)
        inner = (slice(None), slice(p.g, p.g + p.ny), slice(p.g, p.g + p.nx))
        out[inner] = W[inner]
        x = p.x_min + (np.arange(p.nx + 2 * p.g) + 0.5) * (p.x_max - p.x_min) / (p.nx + 2 * p.g)
        right = x > 0.5 * (p.x_min + p.x_max)
        J = float((out[0][:, right] ** 2).sum() * p.dx * p.dy)
        return {"W": out, "J": J, "grad": None}
    p = _problem_2d(case, seed)
    W, U, t, dt = _solve_2d(p, case["steps"])
    if kind == "session":
        W, U = torch.stack(W), torch.stack(U)
    return {"W": W, "U": U, "steps": case["steps"], "t": t, "dt": dt}
