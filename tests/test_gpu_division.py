"""kun::DivFast, the straight-line division of the window regressions, is the
correctly rounded quotient: its reciprocal of every mantissa is the rounded one
(which makes the quotient's last step exact in Markstein's sense), and quotients
are CUDA's own for every divisor with many dividends, and for the divisor whose
mantissa is all ones, which the theorem leaves out, with every dividend."""
import ctypes
import os

import pytest

from kunquant_gb300 import build

SRC = r"""
#include "kun_device.cuh"
typedef unsigned long long u64;
__device__ float f(unsigned mantissa, int exponent) { return __uint_as_float(((unsigned)(127 + exponent) << 23) | mantissa); }
__device__ void check(float a, float b, u64 *n) {
    kun::DivFast div;
    const float q = div(a, b);
    if (!div.ok) { atomicAdd(&n[1], 1ull); return; }
    if (__float_as_uint(q) != __float_as_uint(__fdiv_rn(a, b))) atomicAdd(&n[0], 1ull);
}
__global__ void reciprocals(u64 *n) {
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    for (int e = -60; e < 60; e += 7) {
        const float b = f(m, e);
        if (__float_as_uint(kun::DivFast::reciprocal(b)) != __float_as_uint(__frcp_rn(b))) atomicAdd(&n[0], 1ull);
    }
}
__global__ void divisors(u64 *n) {
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned r = m * 2654435761u + 12345u;
    for (int i = 0; i < 200; i++) {
        r = r * 1664525u + 1013904223u;
        check(f(i < 8 ? (m + i) & 0x7fffff : r >> 9, (int)(r % 120) - 60), f(m, (int)((r >> 5) % 120) - 60), n);
    }
}
__global__ void all_ones(u64 *n) {
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    for (int e = -60; e < 60; e += 17)
        for (int g = -60; g < 60; g += 11) check(f(m, e), f(0x7fffff, g), n);
}
extern "C" __attribute__((visibility("default"))) int division_check(int which, u64 *host) {
    u64 *n;
    if (cudaMalloc((void **)&n, 16) != cudaSuccess) return 1;
    cudaMemset(n, 0, 16);
    void (*kernel)(u64 *) = which == 0 ? reciprocals : which == 1 ? divisors : all_ones;
    kernel<<<(1 << 23) / 256, 256>>>(n);
    const cudaError_t e = cudaMemcpy(host, n, 16, cudaMemcpyDeviceToHost);
    cudaFree(n);
    return (int)e;
}
"""


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["reciprocals", "divisors", "all ones"])
def test_divisions_are_correctly_rounded(which, tmp_path):
    src, lib = tmp_path / "division.cu", str(tmp_path / "division.so")
    src.write_text(SRC)
    build._run([build.NVCC] + build.MODULE_FLAGS + ["-shared", str(src), "-o", lib])
    assert os.path.exists(lib)
    n = (ctypes.c_ulonglong * 2)()
    assert ctypes.CDLL(lib).division_check(["reciprocals", "divisors", "all ones"].index(which), n) == 0
    assert n[0] == 0, (which, n[0])
    assert n[1] == 0 or which == "divisors"   # refused: the ends of the range
