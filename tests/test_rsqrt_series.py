"""The Green kernels' FP64 reciprocal square root (rsqrt_series in
beat_engine_b200/csrc/phase.cuh) on a B200, compiled here from the same header,
against long double and against CUDA's rsqrt().

Bound: half an ulp, 2^-53, of the last addition, and the iteration's next term
5 e^3 / 16 with |e| <= 2^-19.5 from the hardware approximation, 2^-60: together
below 2^-53 (1 + 2^-6).  CUDA documents 1 ulp for rsqrt(double), so the two are
at most 2 ulp apart.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from beat_engine_b200 import build

pytestmark = pytest.mark.gpu
HEADER_DIR = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "beat_engine_b200", "csrc")

SOURCE = r"""
#include "phase.cuh"
__global__ void both_kernel(int n, const double *x, double *y, double *z) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    y[i] = bb::rsqrt_series(x[i]);
    z[i] = rsqrt(x[i]);
}
extern "C" int both(int n, const double *x, double *y, double *z) {
    double *d = nullptr;
    const size_t b = sizeof(double) * (size_t)n;
    if (cudaMalloc(&d, 3 * b) != cudaSuccess) return 1;
    int bad = cudaMemcpy(d, x, b, cudaMemcpyHostToDevice) != cudaSuccess;
    if (!bad) {
        both_kernel<<<(n + 255) / 256, 256>>>(n, d, d + n, d + 2 * (size_t)n);
        bad = cudaMemcpy(y, d + n, b, cudaMemcpyDeviceToHost) != cudaSuccess ||
              cudaMemcpy(z, d + 2 * (size_t)n, b, cudaMemcpyDeviceToHost) != cudaSuccess;
    }
    cudaFree(d);
    return bad;
}
"""


def test_rsqrt_series_within_half_an_ulp(tmp_path):
    src, so = tmp_path / "both.cu", tmp_path / "libboth.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc_path(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I",
                    HEADER_DIR, str(src), "-o", str(so)], check=True)
    rng = np.random.default_rng(1)
    powers = 2.0 ** np.arange(-1022, 1024)
    x = np.concatenate([np.ldexp(rng.uniform(0.5, 1.0, 1 << 20), rng.integers(-1021, 1025, 1 << 20)),
                        rng.uniform(1e-6, 10.0, 1 << 19), powers, np.nextafter(powers, np.inf),
                        np.nextafter(powers[1:], 0.0), [np.finfo(np.float64).max]])
    y, z = np.empty_like(x), np.empty_like(x)
    dp = ctypes.POINTER(ctypes.c_double)
    assert ctypes.CDLL(str(so)).both(len(x), x.ctypes.data_as(dp), y.ctypes.data_as(dp), z.ctypes.data_as(dp)) == 0
    ref = 1 / np.sqrt(x.astype(np.longdouble))
    error = np.abs((y - ref) / ref)
    assert error.max() <= 2.0 ** -53 * (1 + 2.0 ** -6), (float(error.max()), float(x[np.argmax(error)]))
    assert np.max(np.abs(y - z) / np.spacing(z)) <= 2.0
