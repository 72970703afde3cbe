"""GPU: the end of a march of the marching SOR kernel's copies: when march_drain
returns, every copy that was issued has landed in shared memory, whatever the
number of steps and the place in the ring of barriers it began at."""
import ctypes

import pytest

from device_code import compile_cuda

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "k_march.cuh"
using namespace ntcfd;
constexpr int kMost = 8, kWords = 4096;     // steps, words of a step's copy

// Issues `steps` copies as the copying thread does, one per place of the ring (the first place is
// step n0's); earlier phases of the barriers are completed first.
__global__ void drain(const float* src, int n0, int steps, int* wrong) {
    extern __shared__ __align__(16) float buf[];
    __shared__ MarchBars bars;
    for (int q = threadIdx.x; q < kMost * kWords; q += blockDim.x) buf[q] = -1.0f;
    if (threadIdx.x == 0)
        for (int q = 0; q <= kMarchAhead; ++q) mbar_init(bars.full + q, 1u);
    fence_bulk();
    __syncthreads();
    if (threadIdx.x == 0) {
        bool ok = true;
        MarchPos pos(0);
        for (int q = 0; q < n0; ++q, pos.next()) mbar_arrive(bars.full + pos.slot);
        for (int q = 0; q < steps; ++q, pos.next()) {
            // a place of the ring is taken again when its copy has landed
            if (q > kMarchAhead) ok = mbar_wait(bars.full + pos.slot, pos.lap ^ 1u) && ok;
            mbar_expect(bars.full + pos.slot, sizeof(float) * kWords);
            bulk_copy(buf + q * kWords, src + q * kWords, sizeof(float) * kWords, bars.full + pos.slot);
        }
        ok = march_drain(&bars, pos, steps) && ok;
        int bad = ok ? 0 : 1;
        for (int q = max(0, steps - 3); q < steps; ++q)
            for (int w = kWords - 1; w >= 0; w -= 127) bad += buf[q * kWords + w] != src[q * kWords + w];
        *wrong = bad;
    }
}

extern "C" int run(int n0, int steps) {
    float* src;
    int* wrong;
    if (steps > kMost || cudaMallocManaged(&src, sizeof(float) * kMost * kWords) || cudaMallocManaged(&wrong, sizeof(int))) return -1;
    for (int q = 0; q < kMost * kWords; ++q) src[q] = 1.0f + q;
    *wrong = -2;
    const size_t smem = sizeof(float) * kMost * kWords;
    if (cudaFuncSetAttribute(drain, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) return -3;
    drain<<<1, 128, smem>>>(src, n0, steps, wrong);
    const int rc = cudaDeviceSynchronize() ? -4 : *wrong;
    cudaFree(src);
    cudaFree(wrong);
    return rc;
}
"""


def test_no_copy_is_in_flight_after_the_drain(tmp_path):
    lib = compile_cuda(tmp_path, SOURCE)
    lib.run.restype = ctypes.c_int
    for n0 in range(7):
        for steps in range(9):
            assert lib.run(n0, steps) == 0, (n0, steps)
