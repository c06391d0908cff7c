"""Richardson's relaxation factor where no positive number of power-method
steps is given.  Small systems take the default of 30 in both formats (they
did before the one-launch solves took over SELL-32); larger ones form it from
the starting vector alone, in the one-launch solve as in the kernel loop, and
a negative number counts as none."""
import numpy as np
import pytest

import cufoam_gb300 as cf
from cufoam_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _omega(M, n, steps, **opts):
    p = cf.cuFoamRichardson("p", M, {"tolerance": 1e-6, "maxIter": 3, "powerMaxSteps": steps, "reduction": "fast",
                                     **opts}).solve(np.zeros(n), W.uniform(3, n))
    return p.omega


@pytest.mark.parametrize("fmt", ["sell", "csr"])
@pytest.mark.parametrize("box", [(1, 1, 1), (64, 64, 1), (20, 20, 20)])
def test_small_systems_take_the_default(ctx, box, fmt):
    L = W.grid_const(*box, 6.0)
    M = cf.LduMatrix.from_ldu(L, ctx)
    M.set_format(fmt)
    want = _omega(M, L.n, 30)
    assert _omega(M, L.n, 0) == _omega(M, L.n, -1) == want
    M.close()


@pytest.mark.parametrize("box", [(22, 20, 20), (60, 50, 40), (80, 75, 70)])
def test_larger_systems_without_steps(ctx, box):
    L = W.grid_const(*box, 6.0)
    M = cf.LduMatrix.from_ldu(L, ctx)
    M.set_format("sell")
    loop = _omega(M, L.n, 0, useGraph=0)
    one = _omega(M, L.n, 0)
    # (1/n)^2 1' A 1: two sums of n like terms
    assert one == pytest.approx(loop, rel=1e-12) and _omega(M, L.n, -1) == one
    assert one != pytest.approx(_omega(M, L.n, 30), rel=1e-3)
    M.close()
