"""The integer-pipe division and product (csrc/mce_div.cuh) as the GPU runs
them, with the hardware's reciprocal for a seed: the bits of numpy's, over the
operands of the host form's test, for quotients alone, quotients by a shared
divisor, and products."""
import ctypes
import subprocess

import numpy as np
import pytest

from tests.test_division import _operands

pytestmark = pytest.mark.gpu

SRC = """
#include "mce_div.cuh"
__global__ void k(long long n, const double* a, const double* b, double* q)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const mce::DivBy by = mce::div_by(b[i]);
        q[i] = mce::divide(a[i], b[i]);
        q[n + i] = mce::divide(a[i], by);
        q[2 * n + i] = mce::divide(b[n - 1 - i], by);
        q[3 * n + i] = mce::imul(a[i], b[i]);
    }
}
extern "C" int values(long long n, const double* a, const double* b, double* q)
{
    double *da = nullptr, *db = nullptr, *dq = nullptr;
    int bad = cudaMalloc(&da, 8 * n) | cudaMalloc(&db, 8 * n) | cudaMalloc(&dq, 32 * n);
    if (bad) return bad;
    cudaMemcpy(da, a, 8 * n, cudaMemcpyHostToDevice);
    cudaMemcpy(db, b, 8 * n, cudaMemcpyHostToDevice);
    k<<<1024, 256>>>(n, da, db, dq);
    cudaMemcpy(q, dq, 32 * n, cudaMemcpyDeviceToHost);
    cudaFree(da), cudaFree(db), cudaFree(dq);
    return cudaGetLastError();
}
"""


@pytest.mark.parametrize("seed", [5, 6])
def test_quotients_and_products_of_the_device(tmp_path, seed):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cauchyfriendly_gb300 import build
    (tmp_path / "q.cu").write_text(SRC)
    subprocess.run([build._nvcc(), "-shared", str(tmp_path / "q.cu"), "-o", str(tmp_path / "q.so")] + build._flags(),
                   check=True)
    L = ctypes.CDLL(str(tmp_path / "q.so"))
    rng = np.random.Generator(np.random.PCG64(seed))
    n = 4_000_000
    a, b = _operands(rng, n), _operands(rng, n)
    with np.errstate(all="ignore"):
        # dividends a few ulps from a multiple of the divisor: quotients next to a double
        t = (b[: n // 4] * _operands(rng, n // 4)).view(np.uint64) + rng.integers(0, 5, n // 4, dtype=np.uint64)
        a[: n // 4] = (t - np.uint64(2)).view(np.float64)
        want = np.stack([a / b, a / b, b[::-1] / b, a * b])
    got = np.zeros((4, n))
    p = lambda x: x.ctypes.data_as(ctypes.c_void_p)
    assert L.values(ctypes.c_longlong(n), p(a), p(b), p(got)) == 0
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got.view(np.uint64)[~nan], want.view(np.uint64)[~nan])
