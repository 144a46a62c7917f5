"""Performance cases of the sparse-grid DG framework: what a solver program calls in its time loop.

Seven kinds of pass, each through the Python binding's public calls on device state:

  advect         constant-coefficient advection, SSP-RK3 steps on a sparse grid (LinearOperator.rk3_steps)
  burgers_adapt  one whole adaptive Burgers step: predictor, refine, SSP-RK3, coarsen (adaptive_step)
  burgers_steps  SSP-RK3 Burgers steps on a fixed grid (rk3_steps)
  burgers_rhs    one Burgers right-hand side on the caller's vectors (rhs_device)
  wave_adapt     one whole adaptive step of the variable-coefficient wave equation (adaptive_step)
  wave_steps     RK4 wave steps on a fixed grid (rk4_steps)
  batch          SSP-RK3 steps of many independent adaptive advection solves (Batch.rk3_steps)

Each is measured in FP64 and in the mixed precision where it is offered.  `exact` restates the
discretisation in plain 64-bit numpy / torch: dense 1D matrices from piecewise polynomials, transforms
over the fibres of the element set, the adaptive loop on sorted key arrays.

All passes take time steps well below the CFL limit: hundreds of passes of the nonlinear solvers
then stay near the prepared state, whose element count they would otherwise change, and the single
precision part of a mixed step stays small beside the state; the work of a step does not depend on its
length.  Adaptive passes refine below the threshold that the grid
was initialised with, so each step adds elements and coarsens those away that stayed empty, as a
step of a travelling front does.
"""
import functools
import itertools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "adaptive-multiresolution-dg_gb300", "python"))
import amdg  # noqa: E402

SHORT_DT = {"burgers": 2e-7, "wave": 2e-8}
CFL = 0.01  # of the linear cases
ALPHA = 0.825        # LxF constant of the Burgers cases (1.1 times the largest wave speed)
SIGMA, AMP = 10.0, 0.5
REFINE_RATIO = 0.5   # threshold of the adaptive passes over that of the initial grid
COARSEN_RATIO = 0.1  # coarsening threshold over the refinement threshold


def listed():
    return [
        # the smallest solver call: a 2D grid of 5,184 unknowns, one step, launch latency
        {"name": "advect2d_fp64", "path": "advect", "dim": 2, "nmax": 7, "k": 2, "precision": "fp64", "steps": 1},
        # the FP64 production case of four dimensions, 850,176 unknowns
        {"name": "advect4d_fp64", "path": "advect", "dim": 4, "nmax": 8, "k": 2, "precision": "fp64", "steps": 2},
        # cubic elements in five dimensions, blocks of 1,024 coefficients
        {"name": "advect5d_cubic_mixed", "path": "advect", "dim": 5, "nmax": 5, "k": 3, "precision": "mixed", "steps": 2},
        # the largest grid: six dimensions, 34,455,456 unknowns in mixed precision
        {"name": "advect6d_mixed", "path": "advect", "dim": 6, "nmax": 8, "k": 2, "precision": "mixed", "steps": 1},
        # the 2D driver with cubic Hermite interpolation of the flux, a few hundred elements
        {"name": "burgers2d_hermite_adapt", "path": "burgers_adapt", "dim": 2, "nmax": 8, "flux": "hermite",
         "eps": 1e-5, "precision": "fp64"},
        # the 3D adaptive Burgers run that the benchmark reports, about a thousand elements
        {"name": "burgers3d_adapt_fp64", "path": "burgers_adapt", "dim": 3, "nmax": 8, "flux": "lagrange",
         "eps": 1e-5, "precision": "fp64"},
        # the same solver in mixed precision with a tighter threshold
        {"name": "burgers3d_adapt_mixed", "path": "burgers_adapt", "dim": 3, "nmax": 8, "flux": "lagrange",
         "eps": 2e-6, "precision": "mixed"},
        # fixed-grid steps on the 3D sparse grid of 4,096 elements
        {"name": "burgers3d_steps_mixed", "path": "burgers_steps", "dim": 3, "nmax": 8, "precision": "mixed", "steps": 2},
        # one right-hand side for a caller with its own integrator
        {"name": "burgers3d_rhs_fp64", "path": "burgers_rhs", "dim": 3, "nmax": 7, "precision": "fp64"},
        # the adaptive wave equation, some thousands of elements
        {"name": "wave2d_adapt_fp64", "path": "wave_adapt", "nmax": 9, "eps": 1e-7, "precision": "fp64"},
        # wave steps on a filled grid, which the adaptive run tends to (16,384 elements)
        {"name": "wave2d_steps_mixed", "path": "wave_steps", "nmax": 7, "precision": "mixed", "steps": 1},
        # many small independent solves served together
        {"name": "batch3d_mixed", "path": "batch", "solves": 48, "eps": 1e-6, "precision": "mixed", "steps": 2},
    ]


def draw(rng):
    path = rng.choice(["advect", "advect", "burgers_adapt", "burgers_adapt", "burgers_steps", "burgers_rhs",
                       "wave_adapt", "wave_steps", "batch"])
    prec = rng.choice(["fp64", "mixed"])
    log = lambda lo, hi: float("%.3g" % math.exp(rng.uniform(math.log(lo), math.log(hi))))  # noqa: E731
    if path == "advect":
        while True:
            dim, k = rng.randint(2, 6), rng.randint(1, 3)
            nmax = rng.randint(3, 8)
            dof = sparse_size(dim, nmax) * (k + 1) ** dim
            if 500 <= dof <= (3e6 if prec == "fp64" else 2e7) and (k + 1) ** (dim - 1) <= 256:
                break
        return {"path": path, "dim": dim, "nmax": nmax, "k": k, "precision": prec, "steps": rng.randint(1, 4)}
    if path == "burgers_adapt":
        dim = rng.randint(2, 3)
        flux = rng.choice(["lagrange", "hermite"]) if dim == 2 else "lagrange"
        return {"path": path, "dim": dim, "nmax": rng.randint(6, 8), "flux": flux, "eps": log(2e-6, 1e-4),
                "precision": prec}
    if path in ("burgers_steps", "burgers_rhs"):
        dim = rng.randint(2, 3)
        if path == "burgers_rhs":
            return {"path": path, "dim": dim, "nmax": rng.randint(4, 8), "precision": "fp64"}
        return {"path": path, "dim": dim, "nmax": rng.randint(4, 8), "precision": prec, "steps": rng.randint(1, 4)}
    if path == "wave_adapt":
        return {"path": path, "nmax": rng.randint(6, 9), "eps": log(1e-7, 3e-5), "precision": prec}
    if path == "wave_steps":
        return {"path": path, "nmax": rng.randint(4, 7), "precision": prec, "steps": rng.randint(1, 3)}
    return {"path": path, "solves": rng.randint(3, 40), "eps": log(1e-6, 1e-4), "precision": prec,
            "steps": rng.randint(1, 3)}


# ---- what a program has in hand ----------------------------------------------------------------------

_CTX = None


def _context():
    global _CTX
    if _CTX is None:
        _CTX = amdg.Context(0)
    return _CTX


class _Device:
    """n doubles of device memory that belong to `owner`, which lives as long as the tensor made of them."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3}


def _view(owner, ptr):
    """The coefficient vector at ptr of a grid or batch as a tensor, without a copy."""
    return torch.as_tensor(_Device(owner, ptr, owner.dof), device="cuda")


def _data(case, seed):
    """The seed's problem: initial values as separable terms, velocities, thresholds, the time step.

    Where the grid follows the solution, seeds give one element count: they scale the solution with its
    thresholds, reflect it and exchange its axes, which maps the hierarchy to itself."""
    rng = np.random.default_rng([int(seed), 17])
    path, dim = case["path"], case.get("dim", 3 if case["path"] == "batch" else 2)
    if path == "advect":
        phase, amp = rng.uniform(0, 1, dim), rng.uniform(0.5, 2.0)
        vel = rng.uniform(0.3, 1.0, dim) * rng.choice([-1.0, 1.0], dim)
        terms = [lambda x, d: (amp if d == 0 else 1.0) * np.sin(2 * np.pi * (x + phase[d]))]
        return {"terms": terms, "vel": vel, "dt": CFL / (2.0 ** case["nmax"] * np.abs(vel).sum())}
    scale = rng.uniform(0.9, 1.0)
    if path.startswith("burgers"):
        plane = [lambda x, d: np.full_like(x, 0.5 if d == 0 else 1.0)] + _sin_sum(dim, 0.25, 0.3)
        return {"terms": _moved(plane, rng, dim, scale), "eps": scale * case.get("eps", 0.0), "dt": SHORT_DT["burgers"]}
    if path.startswith("wave"):
        # u and u_t move together, in ways that leave the coefficient as it is; u_t as large as a pulse's
        both = [int(rng.integers(0, 2))] * dim, rng.permutation(dim)
        u, v = [_bump(np.array([0.3, 0.4]), 0.07)], [_bump(np.array([0.4, 0.5]), 0.11)]
        return {"terms": _moved(u, rng, dim, scale, both), "velocity": _moved(v, rng, dim, 15.0 * scale, both),
                "eps": scale * case.get("eps", 0.0), "dt": SHORT_DT["wave"]}
    solves, fixed = [], np.random.default_rng(3)
    for _ in range(case["solves"]):
        eps = case["eps"] * math.exp(fixed.uniform(0.0, math.log(10.0)))  # uneven grid sizes
        bumps = [_bump(fixed.uniform(0.2, 0.8, 3), fixed.uniform(0.05, 0.15)) for _ in range(int(fixed.integers(1, 4)))]
        solves.append({"vel": rng.uniform(-1, 1, 3), "eps": scale * eps, "terms": _moved(bumps, rng, 3, scale)})
    return {"solves": solves}


def _moved(terms, rng, dim, scale, moves=None):
    """The sum of the terms times `scale`, reflected in some dimensions, its axes exchanged."""
    flip, axis = (rng.integers(0, 2, dim), rng.permutation(dim)) if moves is None else moves

    def move(f):
        return lambda x, d: (scale if d == 0 else 1.0) * f(1.0 - x if flip[d] else x, axis[d])
    return [move(f) for f in terms]


def _sin_sum(dim, b, c):
    """b sin(2 pi (sum_d x_d + c)) as products of sines and cosines (c in the first factor)."""
    terms = []
    for which in itertools.product((0, 1), repeat=dim):
        n = sum(which)
        if n % 2:
            sign = -1.0 if (n // 2) % 2 else 1.0
            terms.append(lambda x, d, w=which, s=sign: (s * b if d == 0 else 1.0) *
                         (np.sin if w[d] else np.cos)(2 * np.pi * (x + (c if d == 0 else 0.0))))
    return terms


def _bump(centre, width):
    return lambda x, d: sum(np.exp(-((x - centre[d] + m) / width) ** 2) for m in (-1.0, 0.0, 1.0))


def _precision(case):
    return amdg.FP64 if case["precision"] == "fp64" else amdg.MIXED


def _velocity(g, terms, u):
    """u_t of the grid from separable terms; the grid's coefficients stay u."""
    g.init_separable(terms, vectorized=True)
    g.set_velocity(g.coefficients())
    g.set_coefficients(u)


def prepare(case, seed):
    ctx, data, path = _context(), _data(case, seed), case["path"]
    s = {"path": path, "prec": _precision(case), "case": case}
    if path == "advect":
        g = amdg.Grid(ctx, case["dim"], case["nmax"], case["k"])
        g.init_separable(data["terms"], vectorized=True)
        s.update(grid=g, op=amdg.LinearOperator(g, data["vel"]), dt=data["dt"], u=_view(g, g.device_ptr()))
    elif path == "burgers_adapt":
        g = amdg.Grid(ctx, case["dim"], case["nmax"], 2, level_init=3)
        g.init_separable_adaptive(data["terms"], data["eps"], vectorized=True)
        s.update(grid=g, op=amdg.BurgersOperator(g, ALPHA, hermite=case["flux"] == "hermite"), dt=data["dt"])
        s["eps"] = REFINE_RATIO * data["eps"]
    elif path in ("burgers_steps", "burgers_rhs"):
        g = amdg.Grid(ctx, case["dim"], case["nmax"], 2)
        g.init_separable(data["terms"], vectorized=True)
        s.update(grid=g, op=amdg.BurgersOperator(g, ALPHA), dt=data["dt"], u=_view(g, g.device_ptr()))
        if path == "burgers_rhs":
            s["rhs"] = torch.zeros(g.dof, dtype=torch.float64, device="cuda")
    elif path in ("wave_adapt", "wave_steps"):
        if path == "wave_adapt":
            g = amdg.Grid(ctx, 2, case["nmax"], 2, level_init=3)
            g.init_separable_adaptive(data["terms"], data["eps"], vectorized=True)
        else:
            g = amdg.Grid(ctx, 2, case["nmax"], 2, sparse=False)
            g.init_separable(data["terms"], vectorized=True)
        _velocity(g, data["velocity"], g.coefficients())
        s.update(grid=g, op=amdg.WaveOperator(g, SIGMA, AMP), dt=data["dt"], eps=REFINE_RATIO * data["eps"])
    else:
        grids = []
        for w in data["solves"]:
            g = amdg.Grid(ctx, 3, 8, 2, level_init=2)
            g.init_separable_adaptive(w["terms"], w["eps"], vectorized=True)
            grids.append(g)
        batch = amdg.Batch(ctx, grids, [w["vel"] for w in data["solves"]])
        batch.set_dt([_batch_dt(g.max_mesh_level(), w["vel"]) for g, w in zip(grids, data["solves"])])
        s.update(grids=grids, batch=batch, u=_view(batch, _batch_ptr(batch)))
    ctx.synchronize()
    torch.cuda.synchronize()
    return s


def _batch_dt(levels, vel):
    return CFL / float(np.abs(vel) @ (2.0 ** np.asarray(levels)))


def _batch_ptr(batch):
    import ctypes
    p = ctypes.c_void_p()
    if amdg.load().amdg_batch_coefficients_device(batch._h, ctypes.byref(p), None):
        raise RuntimeError("amdg_batch_coefficients_device failed")
    return p.value


def _short_cfl(g, dt):
    """The CFL number that makes an adaptive step dt long on the grid's current finest levels."""
    return dt * float((2.0 ** g.max_mesh_level()).sum())


def run(state):
    s, path, prec = state, state["path"], state["prec"]
    if path == "advect":
        s["op"].rk3_steps(s["dt"], s["case"]["steps"], prec)
        return s["u"]
    if path == "burgers_steps":
        s["op"].rk3_steps(s["dt"], s["case"]["steps"], prec)
        return s["u"]
    if path == "burgers_rhs":
        s["op"].rhs_device(s["u"].data_ptr(), s["rhs"].data_ptr(), prec)
        return s["rhs"]
    if path == "batch":
        s["batch"].rk3_steps(s["case"]["steps"], prec)
        return s["u"]
    g = s["grid"]
    if path == "wave_steps":
        s["op"].rk4_steps(s["dt"], s["case"]["steps"], prec)
        return {"u": _view(g, g.device_ptr()), "u_t": g.velocity()}
    s["op"].adaptive_step(_short_cfl(g, s["dt"]), 1.0, s["eps"], COARSEN_RATIO * s["eps"], prec)
    u = _view(g, g.device_ptr())
    return u if path == "burgers_adapt" else {"u": u, "u_t": g.velocity()}


# ---- the work a pass cannot do without -----------------------------------------------------------------

def sparse_size(dim, nmax):
    """Elements of the sparse grid: level sums up to nmax, 2^(l-1) elements per level l >= 1."""
    per = [1] + [0] * nmax
    for _ in range(dim):
        per = [sum(per[n - l] * (1 if l == 0 else 1 << (l - 1)) for l in range(n + 1)) for n in range(nmax + 1)]
    return sum(per)


@functools.lru_cache(maxsize=None)
def _adaptive_size(path, dim, nmax, eps):
    case = {"path": path, "dim": dim, "nmax": nmax, "solves": 1, "eps": eps}
    data = _data(case, 0)
    w = data["solves"][0] if path == "batch" else data
    return len(_adaptive_set(_Basis(nmax), dim, 2 if path == "batch" else 3, w["terms"], w["eps"])[0])


def work(case):
    """Bytes: the state read and written once per pass.  Flops: 1D transforms over the element's own
    block and, per dimension, its ancestors' and its finer neighbours' blocks (2 * mean level)."""
    path, dim, k = case["path"], case.get("dim", 3 if case["path"] == "batch" else 2), case.get("k", 2)
    if path in ("advect", "burgers_steps", "burgers_rhs"):
        E = sparse_size(dim, case["nmax"])
    elif path == "wave_steps":
        E = 4 ** case["nmax"]
    else:
        E = _adaptive_size(path, dim, case.get("nmax", 8), case["eps"]) * case.get("solves", 1)
    dof, fields = E * (k + 1) ** dim, 2 if path.startswith("wave") else 1
    steps = case.get("steps", 1)
    if path in ("advect", "batch"):
        return {"bytes": 16.0 * dof, "flops": 3.0 * steps * dof * 2 * (k + 1) * dim * 4}
    stages = {"burgers_adapt": 4, "burgers_steps": 3 * steps, "burgers_rhs": 1, "wave_adapt": 4,
              "wave_steps": 4 * steps}[path]
    p1 = 5 if path.startswith("wave") else 4
    sweeps = fields * (1 + dim)  # one transform to the points per field, one back per dimension
    return {"bytes": 16.0 * dof * fields, "flops": 1.0 * stages * E * p1 ** dim * 2 * p1 * dim * sweeps * 8}


# ---- the same results in 64 bits from the definition -----------------------------------------------------
# 1D element orders: 0 for level 0, 2^(n-1) + j for interval j of level n.  A 1D basis function is a
# polynomial on each half of its support, in the support's coordinate in [0, 1].

def _level(o):
    o = np.asarray(o)
    return np.where(o == 0, 0, np.floor(np.log2(np.maximum(o, 1))).astype(np.int64) + 1)


def _polys_alpert(k):
    """(level 0, level >= 1) polynomials, [function][half][power]; the level >= 1 ones by parity."""
    leg = [np.polynomial.Legendre.basis(p, [0, 1]).convert(kind=np.polynomial.Polynomial, domain=[-1, 1]).coef
           * math.sqrt(2 * p + 1) for p in range(k + 1)]
    zero = np.zeros((k + 1, 2, k + 1))
    for p, c in enumerate(leg):
        zero[p, :, :len(c)] = c
    right = {1: [[-1, 2], [-2, 3]], 2: [[1, -24, 30], [3, -16, 15], [4, -15, 12]],
             3: [[1, 4, -30, 28], [-4, 105, -300, 210], [-5, 48, -105, 64], [-16, 105, -192, 105]]}[k]
    one = np.zeros_like(zero)
    for p, c in enumerate(right):  # f(y), y = 2z - 1 >= 0; f(-y) = (-1)^(p+k+1) f(y); unit norm on [0, 1]
        f = np.polynomial.Polynomial(c)
        f = f / math.sqrt(2 * (f * f).integ()(1.0)) * math.sqrt(2.0)
        one[p, 1] = f(np.polynomial.Polynomial([-1, 2])).coef
        one[p, 0] = f(np.polynomial.Polynomial([1, -2])).coef * (-1.0) ** (p + k + 1)
    return zero, one


def _cardinal(nodes, i):
    f = np.polynomial.Polynomial([1.0])
    for m, x in enumerate(nodes):
        if m != i:
            f = f * np.polynomial.Polynomial([-x, 1.0]) / (nodes[i] - x)
    return f.coef


TINY = 1e-13  # the interpolation points sit this far off the element boundaries
# degree: level-0 nodes, their points' shifts, level >= 1 points and shifts, the half of each, half nodes; in [-1, 1]
_LAGRANGE = {
    3: ([-0.6, -0.2, 0.2, 0.6], [0, 0, 0, 0], [-0.8, -0.4, 0.4, 0.8], [0, 0, 0, 0], [0, 0, 1, 1],
        [[-0.8, -0.6, -0.4, -0.2], [0.2, 0.4, 0.6, 0.8]]),
    4: ([-1, -0.5, 0, 0.5, 1], [1, -1, -1, -1, -1], [-0.75, -0.25, 0, 0.25, 0.75], [-1, -1, 1, -1, -1],
        [0, 0, 1, 1, 1], [[-1, -0.75, -0.5, -0.25, 0], [0, 0.25, 0.5, 0.75, 1]]),
}


class _Family:
    """All 1D functions of one basis up to level nmax, evaluated by cell (halves of the finest supports)."""

    def __init__(self, nmax, zero, one, scale):
        self.n1, self.np = 1 << nmax, zero.shape[0]
        o = np.arange(self.n1)
        self.lev = _level(o)
        self.width = np.where(o == 0, 1.0, 2.0 ** -np.maximum(self.lev - 1, 0))
        self.left = np.where(o == 0, 0.0, (o - 2.0 ** np.maximum(self.lev - 1, 0)) * self.width)
        self.coef = np.where((o == 0)[:, None, None, None], zero[None], one[None])
        self.scale = scale(self.lev)  # [n1, np]

    def at(self, x, cell, deriv=0):
        """[n1 * np, points]: the functions' values at x, each from the piece that holds the point `cell` beside it."""
        z, c = [(y[None] - self.left[:, None]) / self.width[:, None] for y in (x, cell)]
        inside, half = (c > 0) & (c < 1), (c > 0.5).astype(np.int64)
        out = np.zeros((self.n1, self.np, len(x)))
        coef = self.coef
        for _ in range(deriv):
            coef = np.concatenate([coef[..., 1:] * np.arange(1, coef.shape[-1]), np.zeros_like(coef[..., :1])], -1)
        idx = np.arange(self.n1)[:, None]
        for p in range(self.np):
            c4 = coef[idx, p, half]  # [n1, points, powers]
            v = np.zeros_like(z)
            for m in range(coef.shape[-1] - 1, -1, -1):
                v = v * z + c4[..., m]
            out[:, p] = np.where(inside, v * self.scale[:, p][:, None] / self.width[:, None] ** deriv, 0.0)
        return out.reshape(self.n1 * self.np, -1)


class _Basis:
    """The Alpert basis of degree k, an interpolation basis (Lagrange degree 3 / 4 or "hermite"), their 1D matrices."""

    def __init__(self, nmax, k=2, interp=None):
        self.nmax, self.k, self.n1 = nmax, k, 1 << nmax
        self.A = _Family(nmax, *_polys_alpert(k), lambda lev: np.repeat(2.0 ** (np.maximum(lev - 1, 0) / 2)[:, None],
                                                                        k + 1, 1))
        gx, gw = np.polynomial.legendre.leggauss(6)
        h = 2.0 ** -nmax
        self.node = np.arange(self.n1) * h
        mid = self.node + h / 2
        self.x = (mid[:, None] + gx * h / 2).ravel()
        self.cell = np.repeat(mid, 6)
        self.w = np.tile(gw * h / 2, self.n1)
        self.before = np.roll(mid, 1)  # the cell left of node i (periodic), its end point
        self.end = np.where(self.node == 0, 1.0, self.node)
        trace = lambda f, d=0: (f.at(self.end, self.before, d), f.at(self.node, mid, d))  # noqa: E731
        a, (al, ar) = self.A.at(self.x, self.cell), trace(self.A)
        ax = self.A.at(self.x, self.cell, 1)
        self.volx = (a * self.w) @ ax.T
        self.ulft, self.urgt = al @ (ar - al).T, ar @ (ar - al).T
        self.jump = self.urgt - self.ulft
        if interp is None:
            return
        self.I, pts, sides, slopes, self.ancestors = self._interp(interp)
        i, (il, ir) = self.I.at(self.x, self.cell), trace(self.I)
        dl, dr = trace(self.A, 1)
        self.lv, self.lvx = (i * self.w) @ a.T, (i * self.w) @ ax.T
        self.lflx, self.ljv = (il + ir) @ (ar - al).T, (ir - il) @ (dl + dr).T
        near = pts + sides * 1e-5 * h  # off the breaks of every piece; 0: no break there
        self.a2p = np.where(slopes[None], self.A.at(pts, near, 1), self.A.at(pts, near))
        self.a2pd = self.A.at(pts, near, 1)
        self.pts = pts

    def _interp(self, kind):
        """(functions, point coordinates, sides, slope dofs, per order the ancestors (order, point, weights))."""
        o = np.arange(self.n1)
        lev, fam = _level(o), None
        if kind == "hermite":
            n = 4
            zero, one = np.zeros((4, 2, 4)), np.zeros((4, 2, 4))
            zero[:, :] = np.array([[1, 0, -3, 2], [0, 0, 3, -2], [0, 1, -2, 1], [0, 0, -1, 1]])[:, None]
            one[0, 0], one[2, 0] = [0, 0, 12, -16], [0, 0, -2, 4]
            one[1, 1], one[3, 1] = [-4, 24, -36, 16], [-2, 8, -10, 4]
            slope = np.array([0, 0, 1, 1])
            scale = lambda l: 2.0 ** (-np.maximum(l - 1, 0)[:, None] * slope)  # noqa: E731
            loc0, side0 = np.array([0.0, 1.0, 0.0, 1.0]), np.array([1, -1, 1, -1])
            loc1, side1 = np.full(4, 0.5), np.array([-1, 1, -1, 1])
        else:
            n0, s0, n1, s1, half, nodes = _LAGRANGE[kind]
            n, slope = len(n0), np.zeros(len(n0), np.int64)
            zero, one = np.zeros((n, 2, n)), np.zeros((n, 2, n))
            for p in range(n):
                zero[p, :] = _cardinal([(y + 1) / 2 for y in n0], p)
                one[p, half[p]] = _cardinal([(y + 1) / 2 for y in nodes[half[p]]], nodes[half[p]].index(n1[p]))
            scale = lambda l: np.ones((len(l), n))  # noqa: E731
            loc0, side0 = (np.array(n0) + 1) / 2, np.array(s0)
            loc1, side1 = (np.array(n1) + 1) / 2, np.array(s1)
        fam = _Family(self.nmax, zero, one, scale)
        loc = np.where((o == 0)[:, None], loc0, loc1)
        side = np.where((o == 0)[:, None], side0, side1)
        pts = fam.left[:, None] + fam.width[:, None] * loc
        # the ancestors of an element: the points of coarser levels strictly inside its support; the surplus of a
        # value subtracts their interpolant, which on the support is the level-0 interpolation scaled to it
        anc = {}
        place = pts + side * TINY * fam.width[:, None] / 2
        for e in range(1, self.n1):
            lo, hi = fam.left[e], fam.left[e] + fam.width[e]
            oa, q = np.nonzero((lev[:, None] < lev[e]) & (place > lo) & (place < hi))
            own = pts[e]
            z = (own - lo) / fam.width[e]
            wt = np.zeros((n, len(oa)))
            for j, (a, b) in enumerate(zip(oa, q)):
                zj = (pts[a, b] - lo) / fam.width[e]
                if kind == "hermite":
                    r = (0 if zj < 0.5 else 1) + 2 * slope[b]
                else:
                    r = int(np.argmin(np.abs(loc0 - zj)))
                for p in range(n):
                    f = np.polynomial.Polynomial(zero[r, 0])
                    wt[p, j] = (f.deriv() if slope[p] else f)(z[p]) * fam.width[e] ** (slope[r] - slope[p])
            anc[e] = (oa, q, wt)
        return fam, pts.ravel(), side.ravel(), np.tile(slope, self.n1) == 1, anc


def _project(basis, terms, dim):
    """[term][d][1D basis]: the terms' factors against the Alpert functions, by Gauss sums on fine cells."""
    gx, gw = np.polynomial.legendre.leggauss(10)
    cells = max(basis.n1, 64)
    mid = (np.arange(cells) + 0.5) / cells
    x = (mid[:, None] + gx / (2 * cells)).ravel()
    a = basis.A.at(x, np.repeat(mid, 10)) * np.tile(gw / (2 * cells), cells)
    return np.array([[a @ np.broadcast_to(f(x, d), x.shape) for d in range(dim)] for f in terms])


def _blocks(orders, coef, k):
    """The element blocks of sum_term prod_d coef[term][d], [E, (k+1)^dim]."""
    E, dim = orders.shape
    out = 0.0
    for term in coef:
        v = np.ones((E, 1))
        for d in range(dim):
            v = (v[:, :, None] * term[d].reshape(-1, k + 1)[orders[:, d]][:, None]).reshape(E, -1)
        out = out + v
    return out


def _pack(orders, nmax):
    key = np.zeros(len(orders), np.int64)
    for d in range(orders.shape[1]):
        key = (key << nmax) | orders[:, d]
    return key


def _unpack(key, dim, nmax):
    return np.stack([(key >> (nmax * (dim - 1 - d))) & ((1 << nmax) - 1) for d in range(dim)], 1)


def _full_or_sparse(dim, nmax, top, sparse=True):
    lev = [lv for lv in itertools.product(range(top + 1), repeat=dim) if not sparse or sum(lv) <= top]
    rows = [np.stack(np.meshgrid(*[np.arange(1 << (l - 1), 1 << l) if l else np.zeros(1, np.int64) for l in lv],
                                 indexing="ij"), -1).reshape(-1, dim) for lv in lev]
    return _unpack(np.sort(_pack(np.concatenate(rows), nmax)), dim, nmax)


def _children(orders, nmax):
    """[(rows that have one, their child)] over dimensions and the two children."""
    got = []
    for d in range(orders.shape[1]):
        o = orders[:, d]
        for c in (0, 1):
            has = (_level(o) < nmax) & ((o > 0) | (c == 1))
            ch = orders[has].copy()
            ch[:, d] = 2 * ch[:, d] + c
            got.append((np.nonzero(has)[0], ch))
    return got


def _refine(orders, nmax, norms, eps):
    """Elements above eps get all their children, then every parent of an element is present."""
    dim = orders.shape[1]
    key = _pack(orders, nmax)
    want = norms > eps
    new = [ch[want[rows]] for rows, ch in _children(orders, nmax)]
    front = np.unique(np.concatenate([_pack(c, nmax) for c in new]))
    front = front[~np.isin(front, key)]
    while len(front):
        key = np.union1d(key, front)
        o = _unpack(front, dim, nmax)
        up = []
        for d in range(dim):
            p = o[o[:, d] > 0].copy()
            p[:, d] //= 2
            up.append(_pack(p, nmax))
        front = np.unique(np.concatenate(up))
        front = front[~np.isin(front, key)]
    return _unpack(key, dim, nmax)


def _coarsen(orders, nmax, norms, eta):
    """The rows that stay: childless elements below eta go (but not the root), until none does."""
    key, keep = _pack(orders, nmax), np.ones(len(orders), bool)
    kids = [(rows, np.searchsorted(key, _pack(ch, nmax)), _pack(ch, nmax)) for rows, ch in _children(orders, nmax)]
    kids = [(r[ok], at[ok]) for r, at, ck in kids for ok in [(at < len(key)) & (key[np.minimum(at, len(key) - 1)] == ck)]]
    small = (norms < eta) & (orders.max(1) > 0)
    while True:
        busy = np.zeros(len(orders), bool)
        for rows, at in kids:
            busy[rows[keep[at]]] = True
        go = keep & small & ~busy
        if not go.any():
            return keep
        keep &= ~go


def _adaptive_set(basis, dim, level_init, terms, eps):
    coef = _project(basis, terms, dim)
    orders = _full_or_sparse(dim, basis.nmax, level_init)
    while True:
        u = _blocks(orders, coef, basis.k)
        more = _refine(orders, basis.nmax, np.linalg.norm(u, axis=1), eps)
        if len(more) == len(orders):
            return orders, u
        orders = more


class _Space:
    """Transforms of element blocks along one dimension, over the pairs of elements in the same fibre."""

    def __init__(self, basis, orders):
        self.b, self.orders, self.dim = basis, orders, orders.shape[1]
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.order = torch.as_tensor(orders, device=self.dev)
        self.pairs, self.mats = [self._fibre_pairs(t) for t in range(self.dim)], {}

    def _fibre_pairs(self, t):
        """(e, s) for every two elements of a fibre along t."""
        o = self.orders.copy()
        own = o[:, t].copy()
        o[:, t] = 0
        _, fibre, count = np.unique(_pack(o, self.b.nmax), return_inverse=True, return_counts=True)
        perm = np.lexsort((own, fibre.ravel()))
        start = np.concatenate([[0], np.cumsum(count)])[:-1]
        n = count[fibre.ravel()[perm]]
        e = np.repeat(perm, n)
        first = np.repeat(start[fibre.ravel()[perm]], n)
        at = np.arange(len(e)) - np.repeat(np.concatenate([[0], np.cumsum(n)])[:-1], n)
        return e, perm[first + at]

    def mat(self, name, matrix, nf, nt):
        """A 1D matrix as blocks by order pair, and per dimension and L / full / U its nonzero element pairs."""
        if name not in self.mats:
            n1 = self.b.n1
            m = matrix.reshape(n1, nf, n1, nt)
            on = (np.abs(m).max((1, 3)) > 1e-13 * np.abs(m).max())
            lev = _level(np.arange(n1))
            lists = []
            for t in range(self.dim):
                e, s = self.pairs[t]
                oe, os = self.orders[e, t], self.orders[s, t]
                lists.append([tuple(torch.as_tensor(v[ok], device=self.dev) for v in (e, s)) for ok in
                              (on[os, oe] & (lev[os] > lev[oe]), on[os, oe], on[os, oe] & (lev[os] <= lev[oe]))])
            self.mats[name] = (torch.as_tensor(np.ascontiguousarray(m.transpose(0, 2, 1, 3)), device=self.dev), lists)
        return self.mats[name]

    def apply(self, x, t, mat, lu=1):
        """x: [E, n_0, .., n_(dim-1)] transformed along t by the pairs of L (0), full (1) or U (2)."""
        m, lists = mat
        e, s = lists[t][lu]
        y = x.movedim(t + 1, 1)
        rest = y.shape[2:]
        y = y.reshape(x.shape[0], y.shape[1], -1)
        out = torch.zeros(x.shape[0], m.shape[3], y.shape[2], dtype=torch.float64, device=self.dev)
        step = max(1, int(5e7) // (y.shape[1] * y.shape[2]))
        for i in range(0, len(e), step):
            ei, si = e[i:i + step], s[i:i + step]
            out.index_add_(0, ei, m[self.order[si, t], self.order[ei, t]].transpose(1, 2) @ y[si])
        return out.reshape(x.shape[0], m.shape[3], *rest).movedim(1, t + 1)

    def chain(self, x, mats):
        """sum over the 2^(dim-1) L / U partial sums of the transforms mats[t], finer parts first."""
        out = 0.0
        for bits in itertools.product((0, 2), repeat=self.dim - 1):
            tags = list(bits) + [1]
            y = x
            for t in sorted(range(self.dim), key=lambda d: (tags[d], d)):
                y = self.apply(y, t, mats[t], tags[t])
            out = out + y
        return out

    def surplus(self, v):
        """Interpolation coefficients from point values: per dimension, minus the coarser levels' interpolant."""
        key = _pack(self.orders, self.b.nmax)
        for d in range(self.dim):
            y = v.movedim(d + 1, 1).reshape(v.shape[0], self.b.I.np, -1)
            out = y.clone()
            for o in np.unique(self.orders[:, d]):
                if o == 0:
                    continue
                oa, q, wt = self.b.ancestors[int(o)]
                rows = np.nonzero(self.orders[:, d] == o)[0]
                for j in range(len(oa)):
                    anc = self.orders[rows].copy()
                    anc[:, d] = oa[j]
                    at = torch.as_tensor(np.searchsorted(key, _pack(anc, self.b.nmax)), device=self.dev)
                    w = torch.as_tensor(wt[:, j].copy(), device=self.dev)
                    out[rows] -= w[None, :, None] * y[at, int(q[j])][:, None]
            v = out.reshape(v.shape[0], self.b.I.np, *v.movedim(d + 1, 1).shape[2:]).movedim(1, d + 1)
        return v

    # right-hand sides of u as [E, (k+1)^dim]
    def _shape(self, u):
        return u.reshape(u.shape[0], *[self.b.k + 1] * self.dim)

    def advect(self, u, vel):
        b, u, n = self.b, self._shape(u), self.b.k + 1
        return sum(self.apply(u, t, self.mat(("advect", t), vel[t] * (b.volx + (b.ulft if vel[t] >= 0 else b.urgt)), n, n))
                   for t in range(self.dim)).reshape(u.shape[0], -1)

    def burgers(self, u):
        b, x, n, P = self.b, self._shape(u), self.b.k + 1, self.b.I.np
        a2p = self.mat("a2p", b.a2p, n, P)
        up = self.chain(x, [a2p] * self.dim)
        if b.I.scale[-1, -1] != 1.0:  # Hermite: value and slopes, f = u^2 / 2, f' = u, f'' = 1
            v = up.reshape(-1, 2, 2, 2, 2)  # slope along 0, point, slope along 1, point
            f, g, h, w = v[:, 0, :, 0], v[:, 1, :, 0], v[:, 0, :, 1], v[:, 1, :, 1]
            fp = torch.stack([torch.stack([f * f / 2, f * h], 2), torch.stack([f * g, g * h + f * w], 2)], 1)
            fp = fp.reshape(up.shape)
        else:
            fp = up * up / 2
        fu = self.surplus(fp)
        lv = self.mat("lv", b.lv, P, n)
        back = self.mat("burgers", b.lvx + 0.5 * b.lflx, P, n)
        pen = self.mat("jump", b.jump, n, n)
        return sum(self.chain(fu, [back if t == d else lv for t in range(self.dim)]) - ALPHA / 2 * self.apply(x, d, pen)
                   for d in range(self.dim)).reshape(u.shape[0], -1)

    def penalty(self, u):
        x, n = self._shape(u), self.b.k + 1
        dx = 2.0 ** -int(_level(self.orders).max())
        pen = self.mat("jump", self.b.jump, n, n)
        return sum(-SIGMA / dx * self.apply(x, d, pen) for d in range(self.dim)).reshape(u.shape[0], -1)

    def wave(self, u):
        b, x, n, P, dim = self.b, self._shape(u), self.b.k + 1, self.b.I.np, self.dim
        a2p, a2pd = self.mat("a2p", b.a2p, n, P), self.mat("a2pd", b.a2pd, n, P)
        sines = torch.as_tensor(np.sin(2 * np.pi * b.pts).reshape(b.n1, P), device=self.dev)
        prod = 1.0
        for d in range(dim):
            prod = prod * sines[self.order[:, d]].reshape(-1, *[P if t == d else 1 for t in range(dim)])
        K = (1 + AMP * prod) ** 2
        lv, ljv = self.mat("lv", b.lv, P, n), self.mat("ljv", b.ljv, P, n)
        back = self.mat("wave", -b.lvx - 0.5 * b.lflx, P, n)
        ku = self.surplus(K * self.chain(x, [a2p] * dim))
        out = self.penalty(u).reshape(x.shape)
        for d in range(dim):
            kx = self.surplus(K * self.chain(x, [a2pd if t == d else a2p for t in range(dim)]))
            out = out + self.chain(kx, [back if t == d else lv for t in range(dim)])
            out = out - 0.5 * self.chain(ku, [ljv if t == d else lv for t in range(dim)])
        return out.reshape(u.shape[0], -1)


def _rk3(f, u, dt, steps):
    for _ in range(steps):
        v = u + dt * f(u)
        v = 3 / 4 * u + 1 / 4 * (v + dt * f(v))
        u = 1 / 3 * u + 2 / 3 * (v + dt * f(v))
    return u


def _rk4(f, u, v, dt, steps):
    """u' = v, v' = f(u)."""
    for _ in range(steps):
        k1, l1 = v, f(u)
        k2, l2 = v + dt / 2 * l1, f(u + dt / 2 * k1)
        k3, l3 = v + dt / 2 * l2, f(u + dt / 2 * k2)
        k4, l4 = v + dt * l3, f(u + dt * k3)
        u, v = u + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4), v + dt / 6 * (l1 + 2 * l2 + 2 * l3 + l4)
    return u, v


def _remap(old, new, nmax, *fields):
    at = torch.as_tensor(np.searchsorted(_pack(new, nmax), _pack(old, nmax)), device=fields[0].device)
    out = [torch.zeros(len(new), f.shape[1], dtype=f.dtype, device=f.device) for f in fields]
    for o, f in zip(out, fields):
        o[at] = f
    return out


def exact(case, seed):
    path, data = case["path"], _data(case, seed)
    if path == "advect":
        b = _Basis(case["nmax"], case["k"])
        s = _Space(b, _full_or_sparse(case["dim"], b.nmax, b.nmax))
        u = torch.as_tensor(_blocks(s.orders, _project(b, data["terms"], s.dim), b.k), device=s.dev)
        return _rk3(lambda v: s.advect(v, data["vel"]), u, data["dt"], case["steps"]).reshape(-1)
    if path == "batch":
        b, out = _Basis(8), []
        if case["solves"] > 16:  # over 20 seconds
            return None
        for w in data["solves"]:
            orders, u = _adaptive_set(b, 3, 2, w["terms"], w["eps"])
            s = _Space(b, orders)
            dt = _batch_dt(_level(orders).max(0), w["vel"])
            out.append(_rk3(lambda v: s.advect(v, w["vel"]), torch.as_tensor(u, device=s.dev), dt,
                            case["steps"]).reshape(-1))
        return torch.cat(out)
    wave = path.startswith("wave")
    dim = case.get("dim", 2)
    b = _Basis(case["nmax"], 2, 4 if wave else "hermite" if case.get("flux") == "hermite" else 3)
    if path.endswith("adapt"):
        orders, u = _adaptive_set(b, dim, 3, data["terms"], data["eps"])
    else:
        orders = _full_or_sparse(dim, b.nmax, b.nmax, sparse=not wave)
        u = _blocks(orders, _project(b, data["terms"], dim), 2)
    s = _Space(b, orders)
    u = torch.as_tensor(u, device=s.dev)
    v = torch.as_tensor(_blocks(orders, _project(b, data["velocity"], dim), 2), device=s.dev) if wave else None
    dt = data["dt"]
    if path == "burgers_rhs":
        return s.burgers(u).reshape(-1)
    if path == "burgers_steps":
        return _rk3(s.burgers, u, dt, case["steps"]).reshape(-1)
    if path == "wave_steps":
        u, v = _rk4(s.wave, u, v, dt, case["steps"])
        return {"u": u.reshape(-1), "u_t": v}
    # the adaptive step: predict, refine on the prediction, step, coarsen
    eps = REFINE_RATIO * data["eps"]
    norm = lambda *f: sum(torch.linalg.norm(x, dim=1) for x in f).cpu().numpy()  # noqa: E731
    predicted = norm(u + dt * v, v + dt * s.penalty(u)) if wave else norm(u + dt * s.burgers(u))
    orders = _refine(s.orders, b.nmax, predicted, eps)
    fields = _remap(s.orders, orders, b.nmax, *([u, v] if wave else [u]))
    s = _Space(b, orders)
    fields = _rk4(s.wave, *fields, dt, 1) if wave else [_rk3(s.burgers, fields[0], dt, 1)]
    keep = torch.as_tensor(_coarsen(orders, b.nmax, norm(*fields), COARSEN_RATIO * eps), device=s.dev)
    fields = [f[keep] for f in fields]
    return {"u": fields[0].reshape(-1), "u_t": fields[1]} if wave else fields[0].reshape(-1)
