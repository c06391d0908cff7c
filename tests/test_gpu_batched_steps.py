"""Batches whose systems take very different numbers of steps: groups of
blocks are sized for like counts, so a system with many more steps must not
be left alone on a few blocks.  Groups pause after a fixed number of steps
and the open systems go on, on all blocks, from their state: the answers are
those of the queue of clusters (other summation orders: counts within a few
percent of the steps), a repeated solve has
the same bits, and the batch takes no longer than on the queue.  A count
beyond several pauses (100, 300, 700 steps), systems that stop at a pause
(maxIter), one and four components, CSR rows among SELL-32 ones."""
import numpy as np
import pytest

from cufoam_gb300 import workloads as W
from cufoam_gb300.batch import BatchSolver

pytestmark = pytest.mark.gpu


def _box(dims, shift, seed):
    L = W.grid_lognormal(*dims, seed)
    return W.LDU(L.n, shift * L.diag, L.lower, L.upper, L.lower_addr, L.upper_addr)


def _uneven(n, seed):
    """Rows too uneven for SELL-32."""
    rng = np.random.default_rng(seed)
    cnt = rng.integers(1, 8, n)
    lo = np.repeat(np.arange(n), cnt)
    hi = lo + rng.integers(1, 60, len(lo))
    pairs = np.unique(np.stack([lo[hi < n], hi[hi < n]], 1), axis=0)
    lo, hi = pairs[:, 0].astype(np.int32), pairs[:, 1].astype(np.int32)
    w = rng.uniform(0.5, 1.5, len(lo))
    d = np.zeros(n)
    np.add.at(d, lo, w)
    np.add.at(d, hi, w)
    return W.LDU(n, 1.0001 * d, -w, -w, lo, hi)


def _systems(count, hard, shift=2.5, lo=8, hi=15, hard_shift=1.0000001):
    rng = np.random.default_rng(count)
    dims = [tuple(int(v) for v in rng.integers(lo, hi, 3)) for _ in range(count)]
    return [_box(d, hard_shift if i in hard else shift, i + 1) for i, d in enumerate(dims)]


def _check_answer(L, b, x, got, first, s, n_rhs):
    """The residual of x is the reported one: every step taken has reached x.
    CG's recurred residual drifts from the true one by the rounding of x and r
    in every step, each below 2^-53 of |A| |x| + |b| (x grows monotonically);
    ten of these per step are allowed.  A step that is missing changes the
    residual by percents."""
    rows = slice(first, first + L.n)
    for j in range(n_rhs):
        v, f = x[rows, j], b[rows, j]
        q = got[s * n_rhs + j]
        r, size = f - L.diag * v, np.abs(f) + np.abs(L.diag * v)
        for i, k, a in ((L.lower_addr, L.upper_addr, L.upper), (L.upper_addr, L.lower_addr, L.lower)):
            np.subtract.at(r, i, a * v[k])
            np.add.at(size, i, np.abs(a * v[k]))
        drift = 10 * (q["n_iterations"] + 1) * 2.0**-53 * np.linalg.norm(size)
        assert abs(np.linalg.norm(r) - q["final_residual"] * q["norm_factor"]) <= drift, (s, j)


@pytest.mark.parametrize("n_rhs", [1, 3, 4])
@pytest.mark.parametrize("precision", ["FP64", "mixed"])
def test_open_systems_go_on_from_their_state(ctx, precision, n_rhs):
    # one system of many steps among easy ones, one of few rows, one in CSR
    systems = _systems(150, {17})
    systems[40] = _box((60, 40, 1), 1.0000001, 3)     # several hundred steps
    systems[41] = _uneven(900, 5)
    systems[42] = _box((3, 2, 1), 2.5, 4)
    B = BatchSolver(systems, n_rhs=n_rhs, context=ctx)
    b = W.uniform(3, n_rhs * B.rows).reshape(B.rows, n_rhs)
    tol = 1e-9
    slack = 0.05 if precision == "FP64" else 0.2      # (FP32 sweeps: the orders differ sooner)
    x, got, _ = B.solve(b, tolerance=tol, max_iter=4000, precision=precision)
    y, want, _ = B.solve(b, tolerance=tol, max_iter=4000, precision=precision, config=(16, 256, 0))
    counts = [q["n_iterations"] for q in want]
    assert min(counts) < 100 and max(counts) > 310     # two pauses at least
    for g, w in zip(got, want):
        assert g["status"] == w["status"] == 0 and g["final_residual"] <= tol
        assert abs(g["n_iterations"] - w["n_iterations"]) <= 2 + slack * w["n_iterations"]
        assert g["initial_residual"] == pytest.approx(w["initial_residual"], rel=1e-12)
        assert g["norm_factor"] == pytest.approx(w["norm_factor"], rel=1e-12)
    for s, L in enumerate(systems):
        _check_answer(L, b, x, got, int(B.offsets[s]), s, n_rhs)
    x2, again, _ = B.solve(b, tolerance=tol, max_iter=4000, precision=precision)
    assert x2.tobytes() == x.tobytes() and again == got
    B.close()


@pytest.mark.parametrize("max_iter", [99, 100, 101, 300, 301])
def test_a_limit_of_steps_around_a_pause(ctx, max_iter):
    systems = _systems(150, {17})
    systems[40] = _box((60, 40, 1), 1.0000001, 3)
    B = BatchSolver(systems, n_rhs=2, context=ctx)
    b = W.uniform(3, 2 * B.rows).reshape(B.rows, 2)
    x, got, _ = B.solve(b, tolerance=1e-9, max_iter=max_iter)
    y, want, _ = B.solve(b, tolerance=1e-9, max_iter=max_iter, config=(16, 256, 0))
    assert max(q["n_iterations"] for q in got) == max_iter
    for g, w in zip(got, want):
        if w["n_iterations"] == max_iter:
            assert g["n_iterations"] == max_iter and g["status"] == w["status"]
        else:
            assert g["status"] == 0 and abs(g["n_iterations"] - w["n_iterations"]) <= 2 + 0.05 * w["n_iterations"]
    for s, L in enumerate(systems):
        _check_answer(L, b, x, got, int(B.offsets[s]), s, 2)
    B.close()


def test_unequal_counts_take_no_longer_than_the_queue(ctx):
    """160 boxes of 12^3..28^3, every twentieth with about five times the steps:
    20.3 ms in groups that were fixed for the whole solve, 13.4 ms on the
    queue of clusters."""
    rng = np.random.default_rng(160)
    dims = [tuple(int(v) for v in rng.integers(12, 29, 3)) for _ in range(160)]
    hard = set(rng.choice(160, 8, replace=False).tolist())
    systems = [_box(d, 1.0000001 if i in hard else 2.5, i + 1) for i, d in enumerate(dims)]
    B = BatchSolver(systems, n_rhs=3, context=ctx)
    b = np.random.default_rng(1).standard_normal((B.rows, 3))
    t = {cfg: min(B.solve(b, tolerance=1e-8, max_iter=5000, config=cfg)[2] for _ in range(5))
         for cfg in ((0, 256, 0), (16, 256, 0))}
    assert t[0, 256, 0] <= 1.25 * t[16, 256, 0], t
    B.close()
