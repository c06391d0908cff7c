"""The work this framework is used for, as measurable cases.

Each case is one call (or one short call sequence) a program makes through
the package's public entry points: a product, a linear solve selected by its
plugin name, a time step with new coefficients in host arrays, the first
solve on a new mesh, a batch of velocity systems, a differentiable solve with
its backward pass.  Systems are the package's own workload generators on
boxes of nx * ny * nz cells:

* "poisson"   constant coefficients with Dirichlet walls (pressure of an
              incompressible flow on a uniform mesh);
* "lognormal" independent face coefficients of strong contrast;
* "momentum"  upwind convection-diffusion plus a transient diagonal term
              (a velocity component, non-symmetric);
* "implicit"  diffusion with a varying (eddy) diffusivity plus a transient
              diagonal term (a scalar transported in time, symmetric).

`numbering` "window" renumbers the cells at random inside windows of 64, the
way an unstructured mesh in a bandwidth-reducing order looks; "shuffled"
renumbers them all.
"""
import math
import types

import numpy as np
import torch

import cufoam_gb300 as cf
from cufoam_gb300 import workloads as W
from cufoam_gb300.autograd import LduPattern, ldu_solve
from cufoam_gb300.batch import BatchSolver


def listed():
    return [
        # y = A x inside a user's own loop (a custom smoother, an operator
        # norm): device vectors, enqueued on the stream
        {"name": "spmv_128", "kind": "spmv", "matrix": "lognormal", "nx": 128, "ny": 128, "nz": 128,
         "numbering": "grid", "row_order": "fast", "transpose": False},
        # a 2-D teaching-size pressure system: latency, nothing else
        {"name": "cg_64x64", "kind": "solve", "solver": "cuFoamCG", "matrix": "poisson", "nx": 64, "ny": 64,
         "nz": 1, "numbering": "grid", "precision": "FP64", "tolerance": 1e-6, "relTol": 0.0, "maxIter": 1000},
        # an inner pressure corrector: a mid-size mesh solved to relTol 0.01
        {"name": "cg_pressure_60", "kind": "solve", "solver": "cuFoamCG", "matrix": "poisson", "nx": 64, "ny": 60,
         "nz": 57, "numbering": "grid", "precision": "FP64", "tolerance": 1e-8, "relTol": 0.01, "maxIter": 1000},
        # the pressure solve of a 2.1-million-cell mesh to 1e-8
        {"name": "cg_poisson_128", "kind": "solve", "solver": "cuFoamCG", "matrix": "poisson", "nx": 128, "ny": 128,
         "nz": 128, "numbering": "grid", "precision": "FP64", "tolerance": 1e-8, "relTol": 0.0, "maxIter": 5000},
        # a velocity component with the default (reference) summation order
        # of BiCG on a renumbered mesh
        {"name": "bicg_momentum_48", "kind": "solve", "solver": "cuFoamBiCG", "matrix": "momentum", "nx": 50, "ny": 48,
         "nz": 47, "numbering": "window", "precision": "FP64", "tolerance": 1e-9, "relTol": 0.0, "maxIter": 1000},
        # the same kind of system on a larger mesh with a diagonally
        # preconditioned minimal-residual iteration
        {"name": "mrjacobi_momentum_96", "kind": "solve", "solver": "cuFoamMRJacobi", "matrix": "momentum", "nx": 100,
         "ny": 96, "nz": 93, "numbering": "grid", "precision": "FP64", "tolerance": 1e-8, "relTol": 0.0,
         "maxIter": 1000},
        # Jacobi sweeps on a mid-size transient scalar
        {"name": "jacobi_implicit_36", "kind": "solve", "solver": "cuFoamJacobi", "matrix": "implicit", "nx": 40,
         "ny": 36, "nz": 33, "numbering": "grid", "precision": "FP64", "tolerance": 1e-8, "relTol": 0.0,
         "maxIter": 1000},
        # FP32 sweeps inside FP64 refinement to a true 1e-10 residual
        {"name": "mixed_cg_implicit_128", "kind": "solve", "solver": "cuFoamCG", "matrix": "implicit", "nx": 128,
         "ny": 128, "nz": 128, "numbering": "grid", "precision": "mixed", "tolerance": 1e-10, "relTol": 0.0,
         "maxIter": 5000},
        # one time step of a solver whose fields live in host memory: new
        # coefficients into the mesh's matrix, then the solve
        {"name": "host_step_80", "kind": "host", "solver": "cuFoamPCG", "matrix": "implicit", "nx": 84, "ny": 80,
         "nz": 77, "numbering": "grid", "tolerance": 1e-8, "relTol": 0.0, "maxIter": 1000},
        # the first solve after the mesh changed: conversion of the
        # addressing on the device, then the solve
        {"name": "new_mesh_56", "kind": "mesh", "solver": "cuFoamPCG", "matrix": "implicit", "nx": 60, "ny": 56,
         "nz": 53, "numbering": "window", "tolerance": 1e-8, "relTol": 0.0, "maxIter": 1000},
        # Ux, Uy, Uz of many uneven subdomains in one launch
        {"name": "batch_velocity_48", "kind": "batch", "systems": 48, "lo": 12, "hi": 36, "n_rhs": 3,
         "numbering": "shuffled", "precision": "FP64", "tolerance": 1e-8, "maxIter": 500},
        # training through a diffusion solve: forward and adjoint
        {"name": "adjoint_diffusion_40", "kind": "adjoint", "nx": 42, "ny": 40, "nz": 39, "tolerance": 1e-12,
         "maxIter": 20000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    return {"nx": _log_int(rng, lo, hi), "ny": _log_int(rng, lo, hi), "nz": _log_int(rng, lo, hi)}


def draw(rng):
    kind = rng.choice(["spmv", "solve", "solve", "solve", "solve", "mixed", "host", "mesh", "batch", "adjoint"])
    if kind == "spmv":
        c = {"kind": "spmv", "matrix": rng.choice(["lognormal", "momentum"]), **_box(rng, 12, 128),
             "numbering": rng.choice(["grid", "grid", "window"]), "row_order": rng.choice(["fast", "fast", "reference"]),
             "transpose": rng.random() < 0.3}
    elif kind in ("solve", "mixed"):
        precision = "mixed" if kind == "mixed" else "FP64"
        solver = rng.choice(["cuFoamCG", "cuFoamMRJacobi"] if kind == "mixed" else
                            ["cuFoamCG", "cuFoamCG", "cuFoamPCG", "cuFoamBiCG", "cuFoamMR", "cuFoamMRJacobi",
                             "cuFoamMRS", "cuFoamJMR", "cuFoamJacobi"])
        if solver == "cuFoamCG" and precision == "FP64":
            matrix = rng.choice(["poisson", "poisson", "implicit"])
        elif solver in ("cuFoamCG", "cuFoamPCG"):
            matrix = "implicit"
        else:
            matrix = rng.choice(["momentum", "momentum", "implicit"])
        box = _box(rng, 10, 120)
        if rng.random() < 0.2:   # a 2-D mesh
            box = {"nx": _log_int(rng, 24, 400), "ny": _log_int(rng, 24, 400), "nz": 1}
        c = {"kind": "solve", "solver": solver, "matrix": matrix, **box,
             "numbering": rng.choice(["grid", "grid", "window"]), "precision": precision,
             "tolerance": 1e-10 if precision == "mixed" else rng.choice([1e-7, 1e-8, 1e-9]),
             "relTol": rng.choice([0.0, 0.01]) if matrix == "poisson" else 0.0, "maxIter": 2000}
    elif kind in ("host", "mesh"):
        c = {"kind": kind, "solver": "cuFoamPCG", "matrix": "implicit", **_box(rng, 12, 88),
             "numbering": "window" if kind == "mesh" else "grid", "tolerance": rng.choice([1e-7, 1e-8]), "relTol": 0.0,
             "maxIter": 1000}
    elif kind == "batch":
        c = {"kind": "batch", "systems": _log_int(rng, 5, 48), "lo": rng.randint(8, 14), "hi": rng.randint(18, 36),
             "n_rhs": rng.choice([1, 2, 3, 3, 4]), "numbering": rng.choice(["grid", "shuffled"]),
             "precision": rng.choice(["FP64", "FP64", "mixed"]), "tolerance": 1e-8, "maxIter": 500}
        if c["precision"] == "mixed":
            c["tolerance"] = 1e-10
    else:
        c = {"kind": "adjoint", **_box(rng, 12, 42), "tolerance": 1e-12, "maxIter": 20000}
    if c.get("numbering") == "window":   # renumbering runs on the host: keep it short
        for k in ("nx", "ny", "nz"):
            c[k] = min(c[k], 72 if c["nz"] > 1 else 300)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _renumber(L, numbering, seed):
    if numbering == "grid":
        return L
    if numbering == "shuffled":
        return W.permute_ldu(L, W.permutation(seed, L.n))
    rng = np.random.default_rng(seed)
    key = np.arange(L.n) // 64 + rng.random(L.n)   # sorting shuffles inside windows of 64
    perm = np.empty(L.n, np.int32)
    perm[np.argsort(key)] = np.arange(L.n, dtype=np.int32)
    return W.permute_ldu(L, perm)


def _implicit(nx, ny, nz, seed):
    """Face diffusivities lognormal(0, 1/4), Dirichlet walls of diffusivity 1
    and a transient term of a quarter of the cell's transport diagonal."""
    L = W.grid_lognormal(nx, ny, nz, seed)
    k = (-L.upper) ** 0.25
    neighbours = np.bincount(L.lower_addr, minlength=L.n) + np.bincount(L.upper_addr, minlength=L.n)
    walls = (6 if nz > 1 else 4) - neighbours
    transport = np.bincount(L.lower_addr, k, L.n) + np.bincount(L.upper_addr, k, L.n) + walls
    L.diag, L.lower, L.upper = 1.25 * transport, -k, -k.copy()
    return L


def _system(c, seed):
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    if c["matrix"] == "poisson":
        L = W.grid_const(nx, ny, nz)
    elif c["matrix"] == "momentum":
        L = W.grid_convdiff(nx, ny, nz, seed, 3.0)[0]
        L.diag = L.diag * 1.25   # the transient term: a quarter of the transport diagonal
    elif c["matrix"] == "implicit":
        L = _implicit(nx, ny, nz, seed)
    else:
        L = W.grid_lognormal(nx, ny, nz, seed)
    return _renumber(L, c["numbering"], seed + 1)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _controls(c):
    return {"solver": c["solver"], "tolerance": c["tolerance"], "relTol": c["relTol"], "maxIter": c["maxIter"],
            "precision": c.get("precision", "FP64")}


def _solver(c, matrix):
    return getattr(cf, c["solver"])("psi", matrix, _controls(c))


def _batch_systems(c, seed):
    u = W.uniform(c["systems"], 3 * c["systems"], 0.0, 1.0).reshape(-1, 3)   # the boxes: the case's, not the seed's
    dims = np.minimum(c["lo"] + (u * (c["hi"] - c["lo"] + 1)).astype(int), c["hi"])
    out = []
    for s, (nx, ny, nz) in enumerate(dims.tolist()):
        L = _implicit(nx, ny, nz, seed + 7 * s + 1)
        out.append(_renumber(L, c["numbering"], seed + 7 * s + 2))
    return out


def prepare(case, seed):
    c, s = dict(case), types.SimpleNamespace(case=dict(case))
    seed = 1000 + 10 * int(seed)
    if c["kind"] == "batch":
        L = _batch_systems(c, seed)
        s.batch = BatchSolver(L, n_rhs=c["n_rhs"])
        s.sources = _dev(W.uniform(seed + 5, s.batch.rows * c["n_rhs"]).reshape(s.batch.rows, c["n_rhs"]))
        return s
    if c["kind"] == "adjoint":
        g = W.grid_grf(c["nx"], c["ny"], c["nz"], seed, 8.0)
        L = W.diffusion_from_cells(c["nx"], c["ny"], c["nz"], g)[0]
        s.pattern = LduPattern(L.n, L.lower_addr, L.upper_addr)
        s.params = [_dev(a).requires_grad_() for a in (L.diag, L.lower, L.upper, W.uniform(seed + 3, L.n))]
        s.target = _dev(W.uniform(seed + 4, L.n, 0.0, 1.0))
        return s
    L = _system(c, seed)
    s.ldu = L
    source = W.uniform(seed + 3, L.n)
    if c["kind"] == "mesh":
        s.source = source
        return s
    s.matrix = cf.LduMatrix.from_ldu(L)
    if c["kind"] == "host":
        s.solver, s.source, s.psi = _solver(c, s.matrix), source, np.empty(L.n)
    elif c["kind"] == "spmv":
        s.x = _dev(source)
        s.y = torch.empty_like(s.x)
        s.matrix.ctx.set_stream(torch.cuda.current_stream())
    else:
        s.solver, s.source = _solver(c, s.matrix), _dev(source)
        s.psi = torch.empty_like(s.source)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    c = s.case
    kind = c["kind"]
    if kind == "spmv":
        return s.matrix.spmv(s.x, transpose=c["transpose"], row_order=c["row_order"], out=s.y)
    if kind == "solve":
        s.psi.zero_()
        perf = s.solver.solve(s.psi, s.source)
        return [s.psi, perf.n_iterations]
    if kind == "host":
        L = s.ldu
        s.psi.fill(0.0)
        s.matrix.update_values(L.diag, L.lower, L.upper)
        perf = s.solver.solve(s.psi, s.source)
        return [s.psi, perf.n_iterations]
    if kind == "mesh":
        matrix = cf.LduMatrix.from_ldu(s.ldu)
        psi = np.zeros(s.ldu.n)
        perf = _solver(c, matrix).solve(psi, s.source)
        matrix.close()
        return [psi, perf.n_iterations]
    if kind == "batch":
        x, res, _ = s.batch.solve(s.sources, tolerance=c["tolerance"], max_iter=c["maxIter"],
                                  precision=c["precision"])
        return [x, np.array([r["n_iterations"] for r in res], np.int32)]
    for p in s.params:
        p.grad = None
    x = ldu_solve(*s.params, s.pattern, {"tolerance": c["tolerance"], "maxIter": c["maxIter"]})
    loss = 0.5 * (x - s.target).square().sum()
    loss.backward()
    return [x.detach(), loss.detach()] + [p.grad for p in s.params]


# ---------------------------------------------------------------------------
# the bytes and operations a pass cannot do without
# ---------------------------------------------------------------------------
def _faces(nx, ny, nz):
    return (nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1)


def _steps(c):
    """Roughly how many steps the iteration takes on these systems."""
    if c["kind"] == "adjoint":
        return 30 * max(c["nx"], c["ny"], c["nz"])
    if c["matrix"] == "poisson":
        return (3.5 if c["relTol"] == 0.0 else 1.5) * max(c["nx"], c["ny"], c["nz"])
    return 40


def work(case):
    c = case
    if c["kind"] == "batch":
        # the mean box, each system's matrix once and its vectors once
        n = c["systems"] * ((c["lo"] + c["hi"]) / 2.0) ** 3
        return {"bytes": n * (7 * 12.0 + 16.0 * c["n_rhs"]), "flops": 25 * c["n_rhs"] * n * 24.0}
    n, f = c["nx"] * c["ny"] * c["nz"], _faces(c["nx"], c["ny"], c["nz"])
    nnz = n + 2 * f
    ldu = 8.0 * (n + 2 * f) + 8.0 * f
    if c["kind"] == "spmv":
        return {"bytes": 8.0 * nnz + 16.0 * n, "flops": 2.0 * nnz}
    steps = _steps(c)
    flops = steps * (2.0 * nnz + 10.0 * n)
    if c["kind"] == "adjoint":
        return {"bytes": 2.0 * ldu + 32.0 * n, "flops": 2.0 * flops}
    if c["kind"] in ("host", "mesh"):
        return {"bytes": ldu + 24.0 * n, "flops": flops}
    matrix = (4.0 if c["precision"] == "mixed" else 8.0) * nnz
    # a matrix larger than the L2 cache is read again in every step
    return {"bytes": matrix * (steps if matrix > 100e6 else 1) + 24.0 * n, "flops": flops}


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------
class _Plain:
    def __init__(self, diag, lower, upper, la, ua):
        self.d, self.lo, self.up = diag, lower, upper
        self.la, self.ua = la.long(), ua.long()

    @classmethod
    def of(cls, L):
        return cls(*(_dev(a) for a in (L.diag, L.lower, L.upper, L.lower_addr, L.upper_addr)))

    def mul(self, x, transpose=False):
        lo, up = (self.up, self.lo) if transpose else (self.lo, self.up)
        y = self.d * x
        y.index_add_(0, self.la, up * x[self.ua])
        return y.index_add_(0, self.ua, lo * x[self.la])

    def norm_factor(self, b):   # psi = 0
        return float(b.norm()) + 1e-20


def _plain_solve(A, b, solver, tolerance, rel_tol, max_iter):
    """The plugin's iteration from psi = 0 in plain torch."""
    x, r = torch.zeros_like(b), b.clone()
    norm0 = norm = float(r.norm())
    tol = max(tolerance * A.norm_factor(b), rel_tol * norm0)
    dinv = 1.0 / A.d
    if solver == "cuFoamJMR":
        sd = dinv.sqrt()
        r = sd * r
        norm0 = norm = float(r.norm())
    k = 0
    if solver in ("cuFoamCG", "cuFoamPCG"):
        z = dinv * r if solver == "cuFoamPCG" else r
        p, rho = z.clone(), float(r @ z)
        while norm > tol and k < max_iter:
            q = A.mul(p)
            a = rho / float(p @ q)
            x += a * p
            r = r - a * q
            norm, k = float(r.norm()), k + 1
            z = dinv * r if solver == "cuFoamPCG" else r
            rho, old = float(r @ z), rho
            p = z + (rho / old) * p
    elif solver == "cuFoamBiCG":
        rs = r.clone()
        p, ps, rho = r.clone(), rs.clone(), float(r @ rs)
        while k < max_iter and (k == 0 or norm >= tol):
            q, qs = A.mul(p), A.mul(ps, True)
            a = rho / float(ps @ q)
            x += a * p
            r, rs = r - a * q, rs - a * qs
            norm, k = float(r.norm()), k + 1
            rho, old = float(r @ rs), rho
            p, ps = r + (rho / old) * p, rs + (rho / old) * ps
    elif solver == "cuFoamJacobi":
        while norm > tol and k < max_iter:
            d = dinv * r
            x += d
            r = r - A.mul(d)
            norm, k = float(r.norm()), k + 1
    else:
        while norm > tol and k < max_iter:
            d = sd * r if solver == "cuFoamJMR" else r if solver == "cuFoamMR" else dinv * r
            y = A.mul(d)
            if solver == "cuFoamJMR":
                y = sd * y
            a = float(r @ y) / float(y @ y)
            x += a * d
            r = r - a * y
            norm, k = float(r.norm()), k + 1
    return x


def exact(case, seed):
    c = dict(case)
    seed = 1000 + 10 * int(seed)
    if c["kind"] == "batch":
        systems = _batch_systems(c, seed)
        rows = sum(L.n for L in systems)
        b = _dev(W.uniform(seed + 5, rows * c["n_rhs"]).reshape(rows, c["n_rhs"]))
        x, at = torch.empty_like(b), 0
        tol = c["tolerance"] if c["precision"] == "FP64" else 1e-13
        for L in systems:
            A = _Plain.of(L)
            for j in range(c["n_rhs"]):
                x[at:at + L.n, j] = _plain_solve(A, b[at:at + L.n, j].contiguous(), "cuFoamCG", tol, 0.0, c["maxIter"])
            at += L.n
        return [x, None]
    if c["kind"] == "adjoint":
        g = W.grid_grf(c["nx"], c["ny"], c["nz"], seed, 8.0)
        L = W.diffusion_from_cells(c["nx"], c["ny"], c["nz"], g)[0]
        A = _Plain.of(L)
        x = _plain_solve(A, _dev(W.uniform(seed + 3, L.n)), "cuFoamCG", c["tolerance"], 0.0, c["maxIter"])
        e = x - _dev(W.uniform(seed + 4, L.n, 0.0, 1.0))
        lam = _plain_solve(A, e, "cuFoamCG", c["tolerance"], 0.0, c["maxIter"])
        return [x, 0.5 * e.square().sum(), -lam * x, -lam[A.ua] * x[A.la], -lam[A.la] * x[A.ua], lam]
    L = _system(c, seed)
    A, b = _Plain.of(L), _dev(W.uniform(seed + 3, L.n))
    if c["kind"] == "spmv":
        return A.mul(b, c["transpose"])
    # a mixed-precision solve ends at its own steps: compared with the solution
    tol = 1e-13 if c.get("precision") == "mixed" else c["tolerance"]
    x = _plain_solve(A, b, c["solver"], tol, c["relTol"], c["maxIter"])
    return [x if c["kind"] == "solve" else x.cpu().numpy(), None]
