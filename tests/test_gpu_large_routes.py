"""Large systems keep the multi-kernel loop where it is the faster form: a
default solve has the bits of the host-driven loop there, in the answer and in
the residuals (the same kernels and sums), and its own sums where it runs as
one launch (Jacobi's answer does not depend on a sum, its residuals do).
Sizes on both sides of the limits (shares of a 135.5 MB L2 taken by 8 bytes per
row, or by the windows of the gathered vector)."""
import numpy as np
import pytest

import cufoam_gb300 as cf
from cufoam_gb300 import workloads as W

pytestmark = pytest.mark.gpu

BOXES = {"160^3": (160, 160, 160), "196^3": (196, 196, 196), "216^3": (216, 216, 216), "3200^2": (3200, 3200, 1)}
# solver, precision -> the boxes that stay one launch
ONE = {("CG", "FP64"): {"160^3", "196^3", "3200^2"}, ("MR", "FP64"): {"160^3", "196^3", "3200^2"},
       ("MRJacobi", "FP64"): {"160^3", "3200^2"}, ("Jacobi", "FP64"): {"160^3", "196^3", "3200^2"},
       ("Richardson", "FP64"): {"160^3"}, ("CG", "mixed"): {"160^3", "196^3", "216^3", "3200^2"},
       ("MR", "mixed"): {"160^3"}, ("MRJacobi", "mixed"): {"160^3"},
       ("BiCG", "mixed"): {"160^3", "196^3", "216^3", "3200^2"}}


@pytest.mark.parametrize("box", BOXES)
def test_the_route_of_large_systems(box):
    ctx = cf.Context(0)
    l2 = 135.5e6
    info = ctx.device_info()
    if not 0.99 * l2 < info["l2_bytes"] < 1.01 * l2:
        pytest.skip("sizes are for another L2")
    G = W.grid_lognormal(*BOXES[box], 5)
    L = W.LDU(G.n, 1.5 * G.diag, G.lower, G.upper, G.lower_addr, G.upper_addr)
    M = cf.LduMatrix.from_ldu(L, ctx)
    b = W.uniform(3, L.n)
    for (name, prec), one in ONE.items():
        out, sums = [], []
        for g in (1, 0):
            x = np.zeros(L.n)
            p = cf._TABLE["cuFoam" + name]("p", M, {"tolerance": 1e-30, "maxIter": 6, "reduction": "fast", "useGraph": g,
                                                    "precision": prec, "powerMaxSteps": 3}).solve(x, b, history=7)
            assert p.n_iterations >= 6 or p.status == 0
            out.append(x)
            sums.append(np.asarray(p.history).tobytes())
        same = out[0].tobytes() == out[1].tobytes() and sums[0] == sums[1]
        assert same == (box not in one), (name, prec)
        # 6 steps of either: the rounding of the sums (FP32 sums within a sweep of mixed)
        assert np.linalg.norm(out[0] - out[1]) <= (1e-12 if prec == "FP64" else 1e-4) * np.linalg.norm(out[1])
    M.close()
    ctx.close()
