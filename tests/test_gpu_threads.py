"""Solves from two host threads, each with its own context: the shared-memory
limit of a kernel belongs to the function on the device, not to a context, so
a solve must never lower it below what another thread is about to launch
with.  The pairs run the same kernel with different amounts of dynamic shared
memory: the matrix in shared memory on the grid, one cluster, the matrix
streamed (vectors alone), mixed precision, the CSR loop's two staging sizes
(fast and reference order), and BiCG.  Every solve returns the bits it
returns alone."""
import threading

import numpy as np
import pytest

import cufoam_gb300 as cf
from cufoam_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _links(n, degree, seed):
    """Diagonally dominant, 1 .. degree forward links per cell at random: rows
    too uneven for SELL-32, staged 256 (degree 4) or 1,024 (degree 9) entries
    at a time."""
    rng = np.random.default_rng(seed)
    cnt = rng.integers(1, degree + 1, n)
    lo = np.repeat(np.arange(n), cnt)
    hi = lo + rng.integers(1, 400, len(lo))
    pairs = np.unique(np.stack([lo[hi < n], hi[hi < n]], 1), axis=0)
    lo, hi = pairs[:, 0].astype(np.int32), pairs[:, 1].astype(np.int32)
    w = rng.uniform(0.5, 1.5, len(lo))
    d = np.ones(n)
    np.add.at(d, lo, w)
    np.add.at(d, hi, w)
    return W.LDU(n, 1.5 * d, -w, -w, lo, hi)


def _box(nx, ny, nz):
    L = W.grid_lognormal(nx, ny, nz, 5)
    return W.LDU(L.n, 1.5 * L.diag, L.lower, L.upper, L.lower_addr, L.upper_addr)


PAIRS = {
    "grid": (lambda: _box(26, 24, 22), lambda: _box(57, 54, 51), "CG", {}),
    "cluster": (lambda: _box(13, 11, 7), lambda: _box(30, 20, 15), "CG", {}),
    "streamed": (lambda: _box(75, 64, 60), lambda: _box(100, 60, 50), "CG", {}),
    "mixed": (lambda: _box(26, 24, 22), lambda: _box(57, 54, 51), "CG", {"precision": "mixed"}),
    "bicg": (lambda: _box(13, 11, 7), lambda: _box(26, 24, 22), "BiCG", {}),
    "csr": (lambda: _links(20000, 4, 1), lambda: _links(20000, 9, 2), "CG", {"useGraph": 0}),
    "csr_reference": (lambda: _links(20000, 4, 1), lambda: _links(20000, 9, 2), "CG",
                      {"useGraph": 0, "reduction": "reference"}),
}


@pytest.mark.parametrize("pair", PAIRS)
def test_two_contexts_solve_at_the_same_time(pair):
    small, large, name, opts = PAIRS[pair]
    start = threading.Barrier(2)
    failures = []

    def work(L):
        ctx = cf.Context(0)
        try:
            M = cf.LduMatrix.from_ldu(L, ctx)
            b = W.uniform(3, L.n)
            S = cf._TABLE["cuFoam" + name]("p", M, {"tolerance": 0.0, "maxIter": 3, **opts})
            want = np.zeros(L.n)
            S.solve(want, b)
            start.wait(60)
            for _ in range(1000):
                x = np.zeros(L.n)
                p = S.solve(x, b)
                if p.status != 1 or x.tobytes() != want.tobytes():   # (1: ended at maxIter)
                    failures.append((L.n, p.status))
                    return
            M.close()
        except Exception as e:   # noqa: BLE001 -- reported by the main thread
            start.abort()
            failures.append((L.n, repr(e)))
        finally:
            ctx.close()

    threads = [threading.Thread(target=work, args=(make(),)) for make in (small, large)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
