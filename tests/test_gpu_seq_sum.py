"""The reference order's sequential sum of block partials, formed by a block
with integer prefix sums: the oracle's bits for sums that change binade
often, cancel, tie on half a unit, span the exponent range or stay at zero,
over one partial, a part of the reference grid and all of it."""
import numpy as np
import pytest

import cufoam_gb300 as cf
import oracle as O

pytestmark = pytest.mark.gpu

RNG = np.random.default_rng(17)
SOURCES = {
    "like": lambda n: RNG.uniform(0.5, 1.5, n),
    "signed": lambda n: RNG.standard_normal(n),
    "integers": lambda n: RNG.integers(-3, 4, n).astype(np.float64),
    "powers": lambda n: np.ldexp(1.0, RNG.integers(-40, 40, n)) * RNG.choice([-1.0, 1.0], n),
    "wide": lambda n: np.ldexp(RNG.uniform(0.5, 1.0, n), RNG.integers(-480, 480, n)),
    "tiny": lambda n: np.ldexp(RNG.uniform(0.5, 1.0, n), -520),
    "sparse": lambda n: np.where(RNG.random(n) < 0.001, RNG.standard_normal(n), 0.0),
    "zero": lambda n: np.zeros(n),
}


@pytest.mark.parametrize("n", [200, 300 * 256 + 5, 1216 * 256 + 77])
@pytest.mark.parametrize("source", list(SOURCES))
def test_reference_order_sums_are_sequential(ctx, ref_grid, source, n):
    L = O.grid_const(n, 1, 1)
    A = O.ldu2csr(L)
    M = cf.LduMatrix.from_ldu(L, ctx)
    b, psi = SOURCES[source](n), SOURCES[source](n)
    assert M.norm_factor(b, psi, reduction="reference") == O.norm_factor(A, b, psi, ref_grid)
    for kind, name in ((O.CG, "cuFoamCG"), (O.BICG, "cuFoamBiCG"), (O.MR, "cuFoamMR")):
        want = O.plugin_solve(kind, L, b, psi.copy(), 1e-300, 4, grid=ref_grid)
        if not np.all(np.isfinite(want.history)):
            continue   # 0/0: the reference goes on with NaN, this library stops (non-finite)
        x = psi.copy()
        perf = cf._TABLE[name]("p", M, {"tolerance": 1e-300, "maxIter": 4, "reduction": "reference"}).solve(
            x, b, history=5)
        assert perf.n_iterations == want.n_iterations
        assert perf.history.tobytes() == want.history.tobytes()
        assert x.tobytes() == want.psi.tobytes()
    M.close()
