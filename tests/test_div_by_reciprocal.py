"""The quotient of a CG step's beta, formed from a reciprocal that is at hand,
against the division it stands for: the function's own source, compiled for
the host with IEEE fused multiply-adds (which CUDA's __fma_rn is).  Quotients
as close to a rounding boundary as 53-bit operands allow, random ones,
exponents up to and beyond the limits of the fast form, zeros, infinities and
NaN: the same bits everywhere."""
import ctypes as C
import os
import random
import re
import struct
import subprocess

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cufoam_gb300", "csrc", "persist.cuh")

SHIM = """
#include <cmath>
#include <cstdint>
#include <cstring>
#define __device__
#define __forceinline__ inline
static int __double2hiint(double v) { uint64_t b; std::memcpy(&b, &v, 8); return (int)(b >> 32); }
static double __dmul_rn(double a, double b) { return a * b; }
static double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
%s
extern "C" void quotients(const double *a, const double *b, double *out, long n)
{
    for (long i = 0; i < n; ++i) {
        const double rb = 1.0 / b[i];
        out[i] = div_by_reciprocal(a[i], b[i], rb);
    }
}
"""


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    text = open(SRC).read()
    i = text.index("__device__ __forceinline__ double div_by_reciprocal(")
    body = text[i:text.index("\n}\n", i) + 3]
    assert re.search(r"__fma_rn\(__fma_rn\(-q, b, a\), rb, q\)", body)
    d = tmp_path_factory.mktemp("div")
    (d / "div.cpp").write_text(SHIM % body)
    so = str(d / "libdiv.so")
    subprocess.check_call(["g++", "-O1", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC", str(d / "div.cpp"),
                           "-o", so])
    lib = C.CDLL(so)

    def run(a, b):
        a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
        out = np.empty_like(a)
        lib.quotients(a.ctypes.data_as(C.c_void_p), b.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p),
                      C.c_long(a.size))
        return out

    return run


def _same(got, a, b):
    with np.errstate(all="ignore"):
        want = a / b
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))


def test_quotients_next_to_a_rounding_boundary(quotients):
    """a = (b N - r) / 2^54 with N odd of 54 bits: a / b is r / (b 2^54) from
    the midpoint of two doubles, the nearest a quotient can come."""
    rnd = random.Random(1)
    a, b = [], []
    while len(a) < 60000:
        k = len(a) % 4
        d = rnd.getrandbits(53) | (1 << 52) | 1 if k < 2 else \
            (1 << 53) - 1 - 2 * rnd.randrange(4000) if k == 2 else (1 << 52) + 1 + 2 * rnd.randrange(4000)
        r = rnd.choice([1, -1, 3, -3, 5, -5])
        n = r * pow(d, -1, 1 << 54) % (1 << 54)
        if n >> 53 == 1 and ((d * n - r) >> 54).bit_length() <= 53:
            a.append(float((d * n - r) >> 54))
            b.append(float(d))
    a, b = np.array(a), np.array(b)
    _same(quotients(a, b), a, b)
    e = np.random.default_rng(2).integers(-800, 700, (2, a.size)).astype(np.int32)
    a, b = np.ldexp(a, e[0]), np.ldexp(-b, e[1])
    _same(quotients(a, b), a, b)


def test_random_and_special_quotients(quotients):
    bits = np.random.default_rng(3).integers(0, 1 << 64, (2, 200000), dtype=np.uint64)
    a, b = bits.view(np.float64)      # every exponent, both signs
    _same(quotients(a, b), a, b)
    special = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2.5e-310, 2.0**-1022, 1.7e308, 1.0, -3.0,
               struct.unpack("d", struct.pack("Q", 200 << 52))[0], struct.unpack("d", struct.pack("Q", 1800 << 52))[0]]
    a, b = [v.ravel() for v in np.meshgrid(special, special)]
    _same(quotients(a, b), a, b)
