"""The device-wide exclusive scans (scan_many) against numpy's cumulative
sums: one launch, two, and the tile sums scanned in between (more than 1,024
tiles of 2,048), with one to four arrays, through the library's own routine."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = """
#include "mce_kernels.cuh"
#include <vector>
// out[j][0..n], total[j]: the scans of in[j][0..n)
extern "C" int scans(const int* in, int jobs, long long n, long long* out, long long* total)
{
    using namespace mce;
    int* di = nullptr;
    long long *dout = nullptr, *tmp = nullptr, *tot = nullptr;
    long long need = 4, t = n;
    while (t > 1) {
        t = (t + 2047) / 2048;
        need += t + 2;
    }
    need = need * kScanJobs + 64;
    int bad = cudaMalloc(&di, sizeof(int) * (jobs * n + 1)) | cudaMalloc(&dout, sizeof(long long) * jobs * (n + 1)) |
              cudaMalloc(&tmp, sizeof(long long) * need) | cudaMallocHost(&tot, sizeof(long long) * jobs);
    if (bad) return bad;
    cudaMemcpy(di, in, sizeof(int) * jobs * n, cudaMemcpyHostToDevice);
    LaunchCfg c{};
    c.num_sms = 152;
    cudaStreamCreate(&c.stream);
    ScanScratch s{tmp, need};
    ScanJob j[kScanJobs];
    for (int k = 0; k < jobs; k++) {
        j[k] = ScanJob{di + k * n, dout + k * (n + 1), k == 1 ? nullptr : tot + k};
        tot[k] = -1;
    }
    scan_many(j, jobs, n, s, c);
    bad = cudaStreamSynchronize(c.stream) | cudaGetLastError();
    cudaMemcpy(out, dout, sizeof(long long) * jobs * (n + 1), cudaMemcpyDeviceToHost);
    for (int k = 0; k < jobs; k++) total[k] = tot[k];
    cudaFree(di), cudaFree(dout), cudaFree(tmp), cudaFreeHost(tot), cudaStreamDestroy(c.stream);
    return bad;
}
"""


@pytest.fixture(scope="module")
def scans(tmp_path_factory):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cauchyfriendly_gb300 import _lib, build
    _lib.load()
    d = tmp_path_factory.mktemp("scan")
    (d / "s.cu").write_text(SRC)
    subprocess.run([build._nvcc(), "-shared", str(d / "s.cu"), "-o", str(d / "s.so"), build.LIB, "-Xlinker",
                    "-rpath=" + build.OUT] + build._flags(), check=True)
    return ctypes.CDLL(str(d / "s.so")).scans


TILES = 1024 * 2048


@pytest.mark.parametrize("jobs", [1, 3, 4])
@pytest.mark.parametrize("n", [0, 1, 2047, 2048, 2049, 6000, TILES - 1, TILES, TILES + 1, 2 * TILES + 12345])
def test_scans_of_every_length(scans, jobs, n):
    rng = np.random.Generator(np.random.PCG64([n, jobs]))
    v = rng.integers(0, 2000, (jobs, n)).astype(np.int32)
    out = np.full((jobs, n + 1), -7, np.int64)
    tot = np.zeros(jobs, np.int64)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert scans(p(v), jobs, ctypes.c_longlong(n), p(out), p(tot)) == 0
    want = np.zeros((jobs, n + 1), np.int64)
    np.cumsum(v, axis=1, out=want[:, 1:])
    assert np.array_equal(out, want)
    for k in range(jobs):
        assert tot[k] == (-1 if k == 1 else want[k, n])
