"""The stopping test of the one-launch solves decides on (r, r) without the
square root unless a history is asked for or the norm is within rounding of
the tolerance: with and without a history, to a tolerance or to a step limit,
a solve takes the same steps and gives the same bits.  One cluster, the matrix
in shared memory, and streamed; tolerances at residuals of the run itself (the
norm within rounding of the tolerance), tolerance 0 and one whose square leaves
the range (the square root is always taken)."""
import numpy as np
import pytest

import cufoam_gb300 as cf
from cufoam_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [(1, 1, 1), (13, 11, 7), (30, 20, 15), (57, 54, 51), (100, 60, 50)])
@pytest.mark.parametrize("name", ["CG", "PCG", "Jacobi", "Richardson", "MR", "MRJacobi", "JMR"])
def test_a_history_does_not_change_the_solve(ctx, name, box):
    G = W.grid_lognormal(*box, 5)
    L = W.LDU(G.n, 1.5 * G.diag, G.lower, G.upper, G.lower_addr, G.upper_addr)
    M = cf.LduMatrix.from_ldu(L, ctx)
    M.set_format("sell")
    b = W.uniform(3, L.n)

    def solve(history, tolerance):
        x = W.uniform(11, L.n, 0.0, 0.5)
        p = cf._TABLE["cuFoam" + name]("p", M, {"reduction": "fast", "maxIter": 30,
                                                    "tolerance": tolerance}).solve(
            x, b, history=31 if history else 0)
        return x, p

    _, run = solve(True, tolerance=1e-30)
    h = np.asarray(run.history)
    nf = run.norm_factor
    at = [float(h[k]) / nf for k in (1, 4, len(h) - 1) if 0 < k < len(h) and h[k] > 0.0]
    near = [v for r in at for v in (r, np.nextafter(r, 0.0), np.nextafter(r, 1e300))]
    for tol in near + [0.0, 1e-30, 1e-170, 1e-6]:
        (x0, p0), (x1, p1) = solve(True, tolerance=tol), solve(False, tolerance=tol)
        assert (p0.n_iterations, p0.status) == (p1.n_iterations, p1.status)
        assert x0.tobytes() == x1.tobytes()
        assert p0.final_residual_abs == p1.final_residual_abs
        if 0 < p1.n_iterations < 30:
            r = np.asarray(p0.history)
            assert r[-1] <= tol * nf and np.all(r[:-1] > tol * nf)
    M.close()
