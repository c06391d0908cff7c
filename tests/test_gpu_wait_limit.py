"""A wait between blocks that runs out: with a limit of one poll some block
gives up at one of a solve's barriers.  Whichever block it is, the solve
returns CF_TIMEOUT (block 0 alone must not decide that), the history holds
only recorded values, and with the default limit the context solves as
before -- the barrier's counter starts from zero again."""
import numpy as np
import pytest

import cufoam_gb300 as cf
from cufoam_gb300 import _capi
from cufoam_gb300 import workloads as W
from cufoam_gb300.batch import BatchSolver

pytestmark = pytest.mark.gpu


def _system(box):
    L = W.grid_lognormal(*box, 5)
    return W.LDU(L.n, 1.5 * L.diag, L.lower, L.upper, L.lower_addr, L.upper_addr)


# the matrix in shared memory, and streamed
@pytest.mark.parametrize("box", [(30, 28, 26), (80, 70, 60)])
@pytest.mark.parametrize("name,opts", [("CG", {}), ("Jacobi", {}), ("MRJacobi", {}), ("BiCG", {}),
                                       ("CG", {"precision": "mixed"}), ("BiCG", {"precision": "mixed"})])
def test_a_wait_that_runs_out_is_a_timeout(box, name, opts):
    ctx = cf.Context(0)
    L = _system(box)
    M = cf.LduMatrix.from_ldu(L, ctx)
    b = W.uniform(3, L.n)
    ctrl = {"tolerance": 1e-9, "maxIter": 400, **opts}
    S = cf._TABLE["cuFoam" + name]("p", M, ctrl)
    x0 = np.zeros(L.n)
    p0 = S.solve(x0, b, history=401)
    assert p0.status == _capi.CF_OK
    for _ in range(3):
        ctx.set_wait_limit(1)
        p = S.solve(np.zeros(L.n), b, history=401)
        assert p.status == _capi.CF_TIMEOUT
        assert 0 <= p.n_iterations <= 400 and len(p.history) <= 401
        ctx.set_wait_limit(0)
        x = np.zeros(L.n)
        p = S.solve(x, b, history=401)
        assert p.status == _capi.CF_OK and p.n_iterations == p0.n_iterations
        assert x.tobytes() == x0.tobytes() and p.history.tobytes() == p0.history.tobytes()
    M.close()
    ctx.close()


@pytest.mark.parametrize("precision", ["FP64", "mixed"])
def test_a_group_of_a_batch_that_runs_out_is_a_timeout(precision):
    ctx = cf.Context(0)
    systems = [_system(b) for b in ((40, 30, 20), (12, 10, 8), (20, 20, 20))]
    B = BatchSolver(systems, n_rhs=2, context=ctx)
    b = W.uniform(3, 2 * B.rows).reshape(B.rows, 2)
    x0, r0, _ = B.solve(b, tolerance=1e-9, max_iter=400, precision=precision)
    ctx.set_wait_limit(1)
    with pytest.raises(cf.CufoamError) as e:
        B.solve(b, tolerance=1e-9, max_iter=400, precision=precision)
    assert e.value.status == _capi.CF_TIMEOUT
    ctx.set_wait_limit(0)
    x, r, _ = B.solve(b, tolerance=1e-9, max_iter=400, precision=precision)
    assert np.array_equal(x, x0) and [q["n_iterations"] for q in r] == [q["n_iterations"] for q in r0]
    B.close()
    ctx.close()


def test_a_negative_limit_is_refused(ctx):
    with pytest.raises(cf.CufoamError):
        ctx.set_wait_limit(-1)
