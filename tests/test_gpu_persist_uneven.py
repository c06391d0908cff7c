"""One-launch solves over meshes whose rows are long in one part of the
numbering and short in another (SELL-32 with the matrix streamed): the blocks
are dealt equal costs, not equal numbers of slices.  The bits of a row do not
depend on its block, so after a fixed number of steps the solves agree with
the host-driven kernel loop to the rounding of the sums, and the time does not
depend on where the long rows are."""
import numpy as np
import pytest

import cufoam_gb300 as cf
from cufoam_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _mesh(n, is_long, width, seed=3):
    """Links from every cell to +1, +a, +b (7-entry rows); cells of is_long
    also to `width` more."""
    a = round(n ** (1 / 3))
    offsets = [1, a, a * a], [2, a - 1, a + 1, a * a + 1, 3, a + 2, 2 * a, a * a - 1][:width]
    lo, hi = [], []
    i = np.arange(n)
    for who, offs in ((i, offsets[0]), (i[is_long], offsets[1])):
        for o in offs:
            c = who[who + o < n]
            lo.append(c)
            hi.append(c + o)
    lo, hi = np.concatenate(lo), np.concatenate(hi)
    order = np.lexsort((hi, lo))
    lo, hi = lo[order].astype(np.int32), hi[order].astype(np.int32)
    w = np.random.default_rng(seed).uniform(0.5, 1.5, len(lo))
    d = np.full(n, 1e-3)
    np.add.at(d, lo, w)
    np.add.at(d, hi, w)
    return W.LDU(n, 1.3 * d, -w, -w, lo, hi)


def _where(n, part):
    i = np.arange(n)
    return {"last": i >= 0.9 * n, "first": i < 0.1 * n, "half": i < 0.5 * n, "few": i < 64}[part]


# 300,000 rows: vectors in shared memory; 1,300,001: partly in global memory, a
# ragged last slice; widths 4 and 8: rows of up to 15 and 23 entries
@pytest.mark.parametrize("n,part,width", [(300000, "last", 4), (300001, "half", 4), (1300001, "first", 4),
                                          (1300001, "last", 8), (300000, "few", 8)])
@pytest.mark.parametrize("name", ["PCG", "Jacobi", "Richardson", "MR", "MRJacobi", "JMR"])
def test_uneven_rows_match_the_kernel_loop(ctx, name, n, part, width):
    L = _mesh(n, _where(n, part), width)
    M = cf.LduMatrix.from_ldu(L, ctx)
    M.set_format("sell")
    b = W.uniform(3, n)
    out = []
    for g in (1, 0):
        psi = W.uniform(11, n, 0.0, 0.5)
        p = cf._TABLE["cuFoam" + name]("p", M, {"useGraph": g, "reduction": "fast", "tolerance": 0.0,
                                                "maxIter": 8}).solve(psi, b, history=9)
        out.append((psi, p))
    (x1, p1), (x0, p0) = out
    assert p1.n_iterations == p0.n_iterations == 8
    # 8 steps, each sum and update a few roundings of 1.1e-16
    assert np.linalg.norm(x1 - x0) <= 1e-13 * np.linalg.norm(x0)
    assert np.allclose(p1.history, p0.history, rtol=1e-11, atol=1e-14 * p0.history[0])
    M.close()


@pytest.mark.parametrize("name", ["CG", "BiCG", "MR"])
def test_uneven_rows_mixed_precision(ctx, name):
    n = 300001
    L = _mesh(n, _where(n, "last"), 8)
    M = cf.LduMatrix.from_ldu(L, ctx)
    b = W.uniform(3, n)
    psi = np.zeros(n)
    p = cf._TABLE["cuFoam" + name]("p", M, {"precision": "mixed", "tolerance": 1e-10, "maxIter": 4000}).solve(psi, b)
    assert p.status == 0 and p.final_residual <= 1e-10
    r = b - L.diag * psi
    np.subtract.at(r, L.lower_addr, L.upper * psi[L.upper_addr])
    np.subtract.at(r, L.upper_addr, L.lower * psi[L.lower_addr])
    # the FP64 residual of the refinement is the true one, to its rounding
    assert np.linalg.norm(r) <= 1.01e-10 * p.norm_factor + 1e-14 * np.linalg.norm(b)
    M.close()


@pytest.mark.parametrize("name", ["CG", "Jacobi"])
def test_the_time_does_not_depend_on_where_the_long_rows_are(ctx, name):
    """A tenth of 2,000,000 rows is long, at the end or in stretches of 1,600
    rows all over the mesh: 60 Jacobi steps took 4.1 ms with equal numbers of
    slices per block and the long rows at the end."""
    n = 2000000
    i = np.arange(n)
    t = {}
    for where, is_long in (("end", i >= 0.9 * n), ("spread", i // 1600 % 10 == 9)):
        M = cf.LduMatrix.from_ldu(_mesh(n, is_long, 4), ctx)
        b = W.uniform(3, n)
        S = cf._TABLE["cuFoam" + name]("p", M, {"tolerance": 0.0, "maxIter": 60})
        t[where] = min(S.solve(np.zeros(n), b).solve_ms for _ in range(5))
        M.close()
    assert t["end"] <= 1.15 * t["spread"], t
