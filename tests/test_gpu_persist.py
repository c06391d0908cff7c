"""The grid-persistent solves (one cooperative launch per solve) against the
host-driven multi-kernel loop: the same arithmetic per row and per element,
only the order of the dot products' partial sums differs, so after a fixed
number of steps the stationary and one-term iterations agree to rounding.
CG, whose steps amplify rounding on systems of strong contrast (ten correct
summation orders of its dot products end the 32 x 20 x 16 system's 67 steps
with final residuals between 7.7e-10 and 9.2e-10), is compared with the
reference algorithm on constant coefficients instead.  Sizes: fewer slices than warps, fewer blocks than SMs, a ragged
last slice, one and several rows per thread, vectors beyond the shared
memory a block may use.  Plus rows summed by the whole warp, the L1
normFactor, min/relTol controls and non-finite input."""
import numpy as np
import pytest

import cufoam_gb300 as cf
import oracle as O
from conftest import assert_fast_order_parity, reference_band
from cufoam_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SOLVERS = ["PCG", "Jacobi", "Richardson", "MR", "MRJacobi", "MRS", "JMR"]
# boxes: 1 row; 33; 1,001 (ragged); 9,000 (one cluster of 16 blocks); 10,240 and
# 10,241 (the last cluster size, the first on the grid); 156,978 (more than one
# row per thread); 300,000 (the matrix streamed, vectors in shared memory);
# 1,300,000 (vectors in global memory)
BOXES = [(1, 1, 1), (33, 1, 1), (13, 11, 7), (30, 20, 15), (32, 20, 16), (77, 19, 7), (57, 54, 51), (100, 60, 50),
         (130, 100, 100)]


def _transient(nx, ny, nz, seed=5):
    """Diffusion of strong contrast with a transient term of half the
    transport diagonal."""
    L = W.grid_lognormal(nx, ny, nz, seed)
    return O.LDU(L.n, L.diag * 1.5, L.lower, L.upper, L.lower_addr, L.upper_addr)


def _pair(M, name, b, opts, history=0):
    out = []
    for g in (1, 0):
        psi = W.uniform(11, b.shape[0], 0.0, 0.5)
        perf = cf._TABLE["cuFoam" + name]("p", M, {"useGraph": g, "reduction": "fast", **opts}).solve(
            psi, b, history=history)
        out.append((psi, perf))
    return out


@pytest.mark.parametrize("box", BOXES)
@pytest.mark.parametrize("name", SOLVERS)
def test_persistent_solve_matches_the_kernel_loop(ctx, name, box):
    L = _transient(*box)
    M = cf.LduMatrix.from_ldu(L, ctx)
    M.set_format("sell")
    b = W.uniform(3, L.n)
    # a history keeps small systems off the single-cluster path
    (x1, p1), (x0, p0) = _pair(M, name, b, {"tolerance": 0.0, "maxIter": 8}, history=9)
    assert p1.n_iterations == p0.n_iterations
    if L.n == 1:     # converges in a step: the residual after it is rounding
        assert np.allclose(x1, x0, rtol=1e-14)
        return
    # 8 steps, each sum and update a few roundings of 1.1e-16
    assert np.linalg.norm(x1 - x0) <= 1e-13 * np.linalg.norm(x0)
    assert np.allclose(p1.history, p0.history, rtol=1e-11, atol=1e-14 * p0.history[0])
    assert abs(p1.norm_factor - p0.norm_factor) <= 1e-14 * p0.norm_factor
    if name == "Richardson":
        assert p1.omega == pytest.approx(p0.omega, rel=1e-13)
    M.close()


@pytest.mark.parametrize("box", BOXES[:-1])
def test_persistent_cg_parity(ctx, box):
    """CG to 1e-9 with a history (small systems included) on constant
    coefficients, where the reference's count does not move under one-ulp
    changes: the count within one, the final residual to 1e-12."""
    L = O.grid_const(*box, diag_value=6.0)
    M = cf.LduMatrix.from_ldu(L, ctx)
    M.set_format("sell")
    b = W.uniform(3, L.n)
    want = O.plugin_solve(O.CG, L, b, np.zeros(L.n), 1e-9, 2000)
    perf = cf.cuFoamCG("p", M, {"tolerance": 1e-9, "maxIter": 2000}).solve(np.zeros(L.n), b, history=2001)
    assert_fast_order_parity(perf, want, reference_band(O.CG, L, b, np.zeros(L.n), 1e-9, 2000, trials=2), 1e-9)


@pytest.mark.parametrize("name", ["MRJacobi"])
def test_persistent_solve_long_rows_and_controls(ctx, name):
    """Rows of up to 300 entries (hub cells) over SELL-32, OpenFOAM's L1
    normFactor, relTol and minIter: the loop's steps and stopping."""
    rng = np.random.default_rng(4)
    n = 12000
    edges = {(i, i + 1) for i in range(n - 1)}
    for h in rng.choice(n // 2, size=12, replace=False):
        edges |= {(int(h), int(j)) for j in rng.choice(np.arange(h + 1, n), size=300, replace=False)}
    e = np.array(sorted(edges), np.int32)
    w = rng.uniform(0.5, 1.5, size=len(e))
    diag = np.ones(n)
    np.add.at(diag, e[:, 0], 1.5 * w)
    np.add.at(diag, e[:, 1], 1.5 * w)
    L = O.LDU(n, diag, -w, -w, e[:, 0].copy(), e[:, 1].copy())
    M = cf.LduMatrix.from_ldu(L, ctx)
    M.set_format("sell")
    b = W.uniform(3, n)
    for opts in ({"tolerance": 1e-9, "normType": "openfoam"}, {"tolerance": 1e-12, "relTol": 0.01},
                 {"tolerance": 10.0, "minIter": 3}):
        (x1, p1), (x0, p0) = _pair(M, name, b, {"maxIter": 500, **opts})
        assert p1.n_iterations == p0.n_iterations and p1.status == p0.status == 0
        assert np.linalg.norm(x1 - x0) <= 1e-12 * np.linalg.norm(x0)
        assert abs(p1.norm_factor - p0.norm_factor) <= 1e-13 * p0.norm_factor


def test_persistent_solve_non_finite_and_reuse(ctx):
    """A NaN in the source stops the solve before its first step; the next
    solve on the same context is unaffected."""
    L = _transient(40, 30, 20)
    M = cf.LduMatrix.from_ldu(L, ctx)
    b = W.uniform(3, L.n)
    want = cf.cuFoamCG("p", M, {"tolerance": 1e-9}).solve(np.zeros(L.n), b)
    bad = b.copy()
    bad[L.n - 1] = np.nan
    p = cf.cuFoamCG("p", M, {"tolerance": 1e-9}).solve(np.zeros(L.n), bad)
    assert p.status == 3 and p.n_iterations == 0
    again = cf.cuFoamCG("p", M, {"tolerance": 1e-9}).solve(np.zeros(L.n), b)
    assert again.n_iterations == want.n_iterations and again.final_residual == want.final_residual
