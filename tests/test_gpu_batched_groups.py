"""Batches of few systems run as groups of blocks, one group per system
(cluster size 0, the default): against the same batch on clusters of four.
Systems of one row, around one slice, with a long row (CSR), randomly
renumbered, and one much larger than the others; 1 to 4 components; one
system alone on the whole device."""
import numpy as np
import pytest

import cufoam_gb300 as cf
import oracle as O
from cufoam_gb300 import workloads as W
from cufoam_gb300.batch import BatchSolver

pytestmark = pytest.mark.gpu


def _transient(L):
    """Face coefficients within a factor of a few and a transient term:
    condition numbers below 100."""
    k = (-L.upper) ** 0.25
    d = np.bincount(L.lower_addr, k, L.n) + np.bincount(L.upper_addr, k, L.n) + 1.0
    return O.LDU(L.n, 1.25 * d, -k, -k, L.lower_addr, L.upper_addr)


def _star(n):
    k = np.full(n - 1, 0.01)
    d = np.ones(n)
    d[0] += k.sum()
    d[1:] += k
    return O.LDU(n, d, -k, -k, np.zeros(n - 1, np.int32), np.arange(1, n, dtype=np.int32))


def _mixed_batch():
    boxes = [(1, 1, 1), (31, 1, 1), (33, 1, 1), (9, 8, 7), (40, 30, 20)]
    out = [_transient(W.grid_lognormal(*b, 3 + i)) for i, b in enumerate(boxes)]
    out[3] = W.permute_ldu(out[3], W.permutation(7, out[3].n))
    return out + [_star(300)]


@pytest.mark.parametrize("n_rhs", [1, 2, 3, 4])
@pytest.mark.parametrize("precision", ["FP64", "mixed"])
def test_groups_match_clusters(ctx, n_rhs, precision):
    systems = _mixed_batch()
    B = BatchSolver(systems, n_rhs=n_rhs, context=ctx)
    rhs = [np.stack([W.uniform(100 * s + j, L.n) for j in range(n_rhs)]) for s, L in enumerate(systems)]
    tol = 1e-11
    kw = dict(tolerance=tol, max_iter=2000, precision=precision)
    xg, rg, _ = B.solve(rhs, **kw)
    xc, rc, _ = B.solve(rhs, config=(4, 256, 0), **kw)
    for a, b, in zip(B.unpack(xg), B.unpack(xc)):
        for j in range(n_rhs):   # both at the tolerance, condition < 100
            assert np.linalg.norm(a[j] - b[j]) <= 2e-9 * np.linalg.norm(b[j])
    for a, b in zip(rg, rc):
        assert a["status"] == b["status"] == 0
        assert abs(a["norm_factor"] - b["norm_factor"]) <= 1e-13 * b["norm_factor"]
        if precision == "FP64":
            assert abs(a["n_iterations"] - b["n_iterations"]) <= 1
    B.close()


@pytest.mark.parametrize("box", [(1, 1, 1), (40, 33, 29), (120, 100, 90)])
def test_one_system_on_the_whole_device(ctx, box):
    L = _transient(W.grid_lognormal(*box, 5))
    B = BatchSolver([L], n_rhs=3, context=ctx)
    b = W.uniform(3, 3 * L.n).reshape(L.n, 3)
    x, res, _ = B.solve(b, tolerance=1e-10, max_iter=500)
    M = cf.LduMatrix.from_ldu(L, ctx)
    for j in range(3):
        r = b[:, j] - M.spmv(np.ascontiguousarray(x[:, j]), row_order="fast")
        assert res[j]["status"] == 0 and np.linalg.norm(r) <= 1.01e-10 * res[j]["norm_factor"]
    x7, res7, _ = B.solve(b, tolerance=1e-14, max_iter=2)   # the step limit
    assert all(q["n_iterations"] <= 2 for q in res7)
    B.close()
    M.close()
