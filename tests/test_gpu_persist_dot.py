"""The dot products of the grid-persistent solves, summed in 64-bit fixed point
per thread, against exact sums: one MR step on a diagonal of powers of two
(the product is exact) returns alpha = (r, A r) / (A r, A r) itself, in a cell
whose source is 1.  Vectors with zeros and subnormals, of one and of both
signs, and of a range beyond 64 bits; sizes of one to several rows per
thread, with remainders (the matrix streamed).

Tolerance: a thread adds at most 2^(head - 1) terms, each cut off below
2^(head - 63) of its largest (head is 5 at the largest size here), which is
below 2^-53 of the sum of magnitudes; the warp, block and grid sums and the
division round once each.  Two sums: below 2^-50, times the cancellation."""
import math

import numpy as np
import pytest

import cufoam_gb300 as cf
import oracle as O

pytestmark = pytest.mark.gpu


def _chain(n, diag):
    z = np.zeros(n - 1)
    return O.LDU(n, diag, z, z.copy(), np.arange(n - 1, dtype=np.int32), np.arange(1, n, dtype=np.int32))


@pytest.mark.parametrize("n", [300000, 600001, 1300001])
@pytest.mark.parametrize("span", [0, 12, 400])
@pytest.mark.parametrize("signs", ["positive", "mixed"])
def test_fixed_point_dots_against_exact_sums(ctx, n, span, signs):
    rng = np.random.default_rng(n + span)
    # 26-bit mantissas: squares are exact
    b = np.ldexp(rng.integers(1, 1 << 26, n).astype(float) * rng.choice([-1.0, 1.0], n), -26)
    b = np.ldexp(b, rng.integers(-span, span + 1, n).astype(np.int32))
    b[::3] = 0.0
    b[1::97] = 5e-310
    b[n // 2] = 1.0
    d = np.ldexp(1.0, rng.integers(-1, 2, n).astype(np.int32))
    if signs == "mixed":
        d *= np.where(rng.random(n) < 0.3, -1.0, 1.0)
    M = cf.LduMatrix.from_ldu(_chain(n, d), ctx)
    M.set_format("sell")
    psi = np.zeros(n)
    perf = cf.cuFoamMR("p", M, {"tolerance": 0.0, "maxIter": 1}).solve(psi, b)
    assert perf.n_iterations == 1 and perf.status == 1     # (ended at maxIter)
    num, mag, den = math.fsum(d * b * b), math.fsum(abs(d) * b * b), math.fsum((d * b) ** 2)
    assert abs(psi[n // 2] - num / den) <= 2.0**-50 * mag / den
    M.close()
