"""The moment chains' parallel exact sums (csrc/mce_chain.cuh) against numpy's
one-after-another sum, bit for bit: series whose sums grow, wander across
binades and zero, cancel, meet halfway values at every step, hold zeros,
infinities or NaN, at lengths around the passes' edges and at odd starts."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = """
#include "mce_chain.cuh"
using namespace mce;
__global__ void k_scan(const double* c, const long long* a, const long long* n, double* o)
{
    __shared__ ChainSmem sm;
    const double s = chain_scan(c, a[blockIdx.x], n[blockIdx.x], sm);
    if (threadIdx.x == 0) o[blockIdx.x] = s;
}
__global__ void k_short(const double* c, const long long* a, const long long* n, double* o)
{
    __shared__ double2 ring[kMomStages][kMomRows / 2][32];
    const double s = chain_short(threadIdx.x == 3 ? c : nullptr, a[blockIdx.x], n[blockIdx.x], ring);
    if (threadIdx.x == 3) o[blockIdx.x] = s;
}
// sums [a[i], a[i] + n[i]) of c[len] into scan[i] and shrt[i]
extern "C" int sums(const double* c, long long len, const long long* a, const long long* n, int cnt, double* scan,
                    double* shrt)
{
    double *dc, *d;
    long long *da, *dn;
    int bad = cudaMalloc(&dc, 8 * len) | cudaMalloc(&d, 16 * cnt) | cudaMalloc(&da, 8 * cnt) | cudaMalloc(&dn, 8 * cnt);
    if (bad) return bad;
    cudaMemcpy(dc, c, 8 * len, cudaMemcpyHostToDevice);
    cudaMemcpy(da, a, 8 * cnt, cudaMemcpyHostToDevice);
    cudaMemcpy(dn, n, 8 * cnt, cudaMemcpyHostToDevice);
    k_scan<<<cnt, kChainThreads>>>(dc, da, dn, d);
    k_short<<<cnt, 32>>>(dc, da, dn, d + cnt);
    cudaMemcpy(scan, d, 8 * cnt, cudaMemcpyDeviceToHost);
    cudaMemcpy(shrt, d + cnt, 8 * cnt, cudaMemcpyDeviceToHost);
    cudaFree(dc), cudaFree(d), cudaFree(da), cudaFree(dn);
    return cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cauchyfriendly_gb300 import build
    d = tmp_path_factory.mktemp("chain")
    (d / "s.cu").write_text(SRC)
    subprocess.run([build._nvcc(), "-shared", str(d / "s.cu"), "-o", str(d / "s.so")] + build._flags(), check=True)
    f = ctypes.CDLL(str(d / "s.so")).sums

    def call(c, a, n):
        c = np.ascontiguousarray(c)
        a, n = np.asarray(a, np.int64), np.asarray(n, np.int64)
        scan, shrt = np.zeros(len(a)), np.zeros(len(a))
        p = lambda x: x.ctypes.data_as(ctypes.c_void_p)
        assert f(p(c), ctypes.c_longlong(len(c)), p(a), p(n), len(a), p(scan), p(shrt)) == 0
        return scan, shrt
    return call


def _series(kind, n, rng):
    if kind == "growing":
        return rng.uniform(0.0, 1.0, n)
    if kind == "wandering":
        return rng.standard_normal(n)
    if kind == "cancelling":  # heavy tails: the sum leaps over binades and comes back
        return rng.standard_cauchy(n) * np.exp(rng.uniform(-30, 2, n))
    if kind == "pairs":  # every large value is taken back by the next
        v = rng.standard_normal(n) * 1e6
        v[1::2] = -v[: n // 2 * 2: 2][: len(v[1::2])] * (1 + 1e-13)
        return v + 1e-9 * rng.standard_normal(n)
    if kind == "halfway":  # on a sum in [1, 2): odd multiples of half its ulp, ties of either parity
        v = rng.integers(-9, 10, n) * 2.0 ** -53
        v[0] = 1.5
        return v
    if kind == "families":  # groups that cancel to rounding noise, of very different sizes
        v = rng.standard_normal(n) * 10.0 ** np.repeat(rng.uniform(-14, 1, n // 6 + 1), 6)[:n]
        v[5::6] = -sum(v[i::6][: len(v[5::6])] for i in range(5))
        return v
    if kind == "zeros":
        v = np.where(rng.integers(0, 50, n) == 0, rng.standard_normal(n), 0.0)
        v[: n // 3] = -0.0
        return v
    v = rng.standard_normal(n) * 1e-300  # tiny, then not finite
    v[n // 2] = np.inf
    v[n // 2 + n // 4] = -np.inf if kind == "nan" else 1.0
    return v


@pytest.mark.parametrize("kind", ["growing", "wandering", "cancelling", "pairs", "families", "halfway", "zeros", "infinite", "nan"])
def test_chain_sums_are_the_sequential_sums(sums, kind):
    rng = np.random.Generator(np.random.PCG64(3))
    v = _series(kind, 60000, rng)
    lens = [1, 2, 7, 8, 9, 63, 64, 65, 1023, 1024, 1025, 2048, 3071, 3073, 4096, 20001, 59000]
    a, n = [0] * len(lens), list(lens)
    a += [int(x) for x in rng.integers(0, 900, len(lens))]  # odd starts among them
    n += lens
    scan, shrt = sums(v, a, n)
    with np.errstate(invalid="ignore", over="ignore"):
        want = np.array([np.add.accumulate(v[i:i + k])[-1] if v[i] != 0 else np.add.accumulate(np.r_[0.0, v[i:i + k]])[-1]
                         for i, k in zip(a, n)])
    for got in (scan, shrt):
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(got), nan)
        assert np.array_equal(got.view(np.int64)[~nan], want.view(np.int64)[~nan]), \
            [(i, k) for i, k, g, w in zip(a, n, got, want) if g != w][:4]
