"""The kernels' integer-pipe division and product (csrc/mce_div.cuh) compiled
for the host: the same bits as IEEE's, the division for seeds an ulp either
side of the correctly rounded single-precision reciprocal (the hardware's is
within one), over random operands and the edges where a digit or the rounding
can go wrong."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cauchyfriendly_gb300", "csrc")

SRC = """
#include "mce_div.cuh"
extern "C" void quotients(long n, const double* a, const double* b, double* q)
{
    for (long i = 0; i < n; i++) q[i] = mce::divide(a[i], b[i]);
}
extern "C" void products(long n, const double* a, const double* b, double* q)
{
    for (long i = 0; i < n; i++) q[i] = mce::imul(a[i], b[i]);
}
"""


def _operands(rng, n):
    """Significands: random, and within 8 of either end, with short tails; exponents around 1, and any."""
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    near = rng.integers(0, 8, n, dtype=np.uint64)
    kind = rng.integers(0, 8, n)
    m = np.where(kind == 1, near, m)
    m = np.where(kind == 2, np.uint64((1 << 52) - 1) - near, m)
    m = np.where(kind == 3, m & ~np.uint64((1 << 29) - 1), m)  # exact in single precision: the seed's own steps
    e = rng.integers(1023 - 60, 1023 + 60, n).astype(np.uint64)
    wide = rng.integers(0, 8, n) == 0
    e = np.where(wide, rng.integers(0, 2048, n).astype(np.uint64), e)  # zeros, subnormals, infinities, NaN too
    m = np.where(wide & (kind >= 6), np.uint64(0), m)
    s = rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63)
    return (s | (e << np.uint64(52)) | m).view(np.float64)


@pytest.mark.parametrize("ulps", [-1, 0, 1])
def test_quotients_and_products_are_the_ieee_ones(tmp_path, ulps):
    src, lib = tmp_path / "q.cpp", tmp_path / "q.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-I" + CSRC,
                    "-DMCE_DIV_SEED_ULPS=(%d)" % ulps, str(src), "-o", str(lib)], check=True)
    L = ctypes.CDLL(str(lib))
    rng = np.random.Generator(np.random.PCG64(5))
    n = 1_000_000
    a, b = _operands(rng, n), _operands(rng, n)
    with np.errstate(all="ignore"):
        # dividends a few ulps from a multiple of the divisor: quotients next to a double
        t = (b[: n // 4] * _operands(rng, n // 4)).view(np.uint64) + rng.integers(0, 5, n // 4, dtype=np.uint64)
        a[: n // 4] = (t - np.uint64(2)).view(np.float64)
        want = a / b
        prod = a * b
    dp = ctypes.POINTER(ctypes.c_double)
    for f, want in ((L.quotients, want), (L.products, prod)):
        got = np.zeros(n)
        f(ctypes.c_long(n), a.ctypes.data_as(dp), b.ctypes.data_as(dp), got.ctypes.data_as(dp))
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(got), nan)
        assert np.array_equal(got.view(np.uint64)[~nan], want.view(np.uint64)[~nan])
