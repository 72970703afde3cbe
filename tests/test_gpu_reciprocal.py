"""GPU: the reciprocals that sweeps form from the coefficient sum (rdiag_near,
and the marching kernel's march_rd) equal the correctly rounded ones bit for
bit: in FP32 for every significand at several exponents, in FP64 for seeded
random significands, the powers of two and their neighbours, and the smallest
and largest sums whose reciprocal is normal."""
import ctypes

import pytest

from device_code import compile_cuda

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "k_march.cuh"
using namespace ntcfd;

__global__ void k32(int exponent, unsigned long long* bad) {
    const unsigned int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= 1u << 23) return;
    const float s = __uint_as_float(((unsigned int)(exponent + 127) << 23) | m), want = __frcp_rn(s);
    const float o = __uint_as_float(((unsigned int)(exponent + 127) << 23) | (m ^ 0x2aaaaau));
    // the marching kernel's sums carry the coefficients' sign
    const Rows<float> two = march_rd(Rows<float>::of(-s, -o));
    const bool ok = rdiag_near(s) == want && two.get(0) == want && two.get(1) == __frcp_rn(o);
    if (!ok) atomicAdd(bad, 1ull);
}

__device__ bool right64(double s) {
    const double want = __drcp_rn(s);
    return rdiag_near(s) == want && march_rd(Rows<double>{s}).v == want;
}

// the exponents -1000 .. 999 with significands near both ends; `each` random ones per thread
__global__ void k64(unsigned long long seed, int each, unsigned long long* bad) {
    const unsigned long long id = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    unsigned long long n = 0ull;
    if (id < 2000ull)
        for (unsigned long long q = 0; q < 64ull; ++q) {
            const unsigned long long e = (id + 23ull) << 52;
            n += !right64(__longlong_as_double((long long)(e | q)));
            n += !right64(__longlong_as_double((long long)(e | (0xfffffffffffffull - q))));
        }
    unsigned long long z = seed + id * 0x9e3779b97f4a7c15ull;
    for (int q = 0; q < each; ++q) {
        z += 0x632be59bd9b4e019ull;
        unsigned long long x = z;
        x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
        x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
        x ^= x >> 31;
        n += !right64(__longlong_as_double((long long)((x >> 12) | ((unsigned long long)(1000 + (int)(x & 63)) << 52))));
    }
    if (n) atomicAdd(bad, n);
}

extern "C" long long run32(int exponent) {
    unsigned long long* bad;
    if (cudaMallocManaged(&bad, sizeof *bad)) return -1;
    *bad = 0ull;
    k32<<<(1 << 23) / 256, 256>>>(exponent, bad);
    const long long r = cudaDeviceSynchronize() ? -2 : (long long)*bad;
    cudaFree(bad);
    return r;
}
extern "C" long long run64(unsigned long long seed, int each) {
    unsigned long long* bad;
    if (cudaMallocManaged(&bad, sizeof *bad)) return -1;
    *bad = 0ull;
    k64<<<148 * 8, 256>>>(seed, each, bad);
    const long long r = cudaDeviceSynchronize() ? -2 : (long long)*bad;
    cudaFree(bad);
    return r;
}
"""


def test_formed_reciprocals_round_to_nearest(tmp_path):
    lib = compile_cuda(tmp_path, SOURCE)
    lib.run32.restype = lib.run64.restype = ctypes.c_longlong
    lib.run64.argtypes = [ctypes.c_ulonglong, ctypes.c_int]
    for exponent in (-100, -37, -1, 0, 1, 17, 100):
        assert lib.run32(exponent) == 0, exponent
    for seed in range(4):
        assert lib.run64(0x123456789 * (seed + 1), 20000) == 0, seed
