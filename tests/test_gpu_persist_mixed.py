"""Mixed-precision solves as one cooperative launch: the FP64 tolerance on the
true residual at sizes where the schedule changes (one block, one cluster,
the first size on the grid, the matrix in shared memory and streamed, vectors
beyond shared memory), the answer against an FP64 solve, and the controls of
the refinement loop."""
import numpy as np
import pytest

import cufoam_gb300 as cf
import oracle as O
from cufoam_gb300 import workloads as W

pytestmark = pytest.mark.gpu

BOXES = [(1, 1, 1), (33, 1, 1), (13, 11, 7), (32, 20, 16), (77, 19, 7), (57, 54, 51), (110, 70, 60), (140, 130, 120)]


def _system(name, box):
    """Transient systems: diffusion for CG, upwind convection-diffusion else."""
    if name == "CG":
        L = W.grid_lognormal(*box, 5)
        k = (-L.upper) ** 0.25          # diffusivities within a factor of a few
        d = np.bincount(L.lower_addr, k, L.n) + np.bincount(L.upper_addr, k, L.n) + 1.0
        return O.LDU(L.n, 1.25 * d, -k, -k, L.lower_addr, L.upper_addr)
    L = W.grid_convdiff(*box, 5, 3.0)[0]
    return O.LDU(L.n, 1.25 * L.diag, L.lower, L.upper, L.lower_addr, L.upper_addr)


@pytest.mark.parametrize("box", BOXES)
@pytest.mark.parametrize("name", ["CG", "MR", "MRJacobi", "JMR", "BiCG"])
def test_mixed_persistent_reaches_the_tolerance(ctx, name, box):
    L = _system(name, box)
    M = cf.LduMatrix.from_ldu(L, ctx)
    M.set_format("sell")
    b = W.uniform(3, L.n)
    tol = 1e-10
    psi = np.zeros(L.n)
    opts = {"tolerance": tol, "maxIter": 5000, "precision": "mixed"}
    perf = cf._TABLE["cuFoam" + name]("p", M, opts).solve(psi, b, history=64)
    if L.n == 33:
        # a badly conditioned row of cells: plain MR stalls there; whatever the
        # kernel loop reaches within the limit, this reaches
        loop = cf._TABLE["cuFoam" + name]("p", M, {**opts, "useGraph": 0}).solve(np.zeros(L.n), b)
        assert perf.status == loop.status, (perf, loop)
        if perf.status != 0:
            assert perf.n_iterations == loop.n_iterations == 5000
            assert 0.5 <= perf.final_residual / loop.final_residual <= 2.0
            return
    assert perf.status == 0 and perf.final_residual <= tol
    assert perf.history.shape[0] == perf.n_outer + 1
    r = b - M.spmv(psi, row_order="fast")
    if name == "JMR":
        r = r / np.sqrt(L.diag)
    assert np.linalg.norm(r) / perf.norm_factor <= tol * (1 + 1e-5)
    # the boxes with cells in all three directions have condition numbers
    # below 100; the row of 33 cells has 510
    if L.n != 33:
        x = np.zeros(L.n)
        cf.cuFoamMRJacobi("p", M, {"tolerance": 1e-13, "maxIter": 5000, "reduction": "fast"}).solve(x, b)
        assert np.linalg.norm(psi - x) <= 1e-8 * np.linalg.norm(x)
    M.close()


def test_mixed_persistent_controls(ctx):
    """relTol ends the refinement early, maxIter bounds the FP32 steps,
    innerMaxIter the steps of a sweep; an answer at the start takes none."""
    L = _system("CG", (30, 28, 26))
    M = cf.LduMatrix.from_ldu(L, ctx)
    b = W.uniform(3, L.n)
    solve = lambda o, x: cf.cuFoamCG("p", M, {"precision": "mixed", "maxIter": 500, **o}).solve(x, b)
    p = solve({"tolerance": 1e-12, "relTol": 1e-3}, np.zeros(L.n))
    assert p.status == 0 and p.n_outer == 1 and p.final_residual <= 1e-3 * p.initial_residual
    p = solve({"tolerance": 1e-12, "maxIter": 7}, np.zeros(L.n))
    assert p.status == 1 and p.n_iterations <= 7
    x = np.zeros(L.n)
    p = solve({"tolerance": 1e-10, "innerMaxIter": 9}, x)
    assert p.status == 0 and p.n_outer >= 3 and p.n_iterations <= 9 * p.n_outer
    q = solve({"tolerance": 1e-9}, x)
    assert q.status == 0 and q.n_iterations == 0
