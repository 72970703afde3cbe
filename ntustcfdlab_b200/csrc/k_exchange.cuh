// k_exchange.cuh -- values handed from CTA to CTA of a cooperative launch without a
// barrier, and verdict counters, for the resident SOR kernel.
//
// A value travels in one atomic word beside a sequence number: the receiver polls
// the word itself, so a hand-over costs one trip through L2 and no flag, fence or
// grid barrier.  Every poll is bounded: a wait that gives up sets the error flag,
// which the other CTAs see in their own waits.
#pragma once

#include "k_gridbar.cuh"
#include "ntcfd_common.cuh"

namespace ntcfd {

constexpr unsigned int kRingPolls = 4000000u;    // polls of one word before giving up (seconds)

// Device memory of the exchange (one per context).  k_defect zeroes all but seq.
struct ResSync {
    GridBar bar;                     // the grid barrier's words, the error flag
    unsigned long long cnt[2][4];    // [colour][sweep & 3]: arrivals, and verdicts in the high half
    unsigned long long last;         // max |change| of the last sweep
    unsigned int seq;                // sequence number of the last half-sweep of earlier launches
    unsigned int pad;
};

// Part b of n rows cut into nb parts whose sizes differ by at most one.
__host__ __device__ inline int brick_start(int b, int n, int nb) { return (int)((long long)b * n / nb); }

// A ring value and its sequence number in one atomic access (two for FP64:
// each half of the double carries the number).
template <class Tc>
struct RingWord;
template <>
struct RingWord<float> {
    static constexpr int n = 1;
    unsigned long long w;
    __device__ __forceinline__ void load(const unsigned long long* p) {
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    }
    __device__ __forceinline__ bool has(unsigned int seq) const { return (unsigned int)(w >> 32) == seq; }
    __device__ __forceinline__ float value() const { return __uint_as_float((unsigned int)w); }
    static __device__ __forceinline__ void store(unsigned long long* p, float v, unsigned int seq) {
        const unsigned long long w = __float_as_uint(v) | ((unsigned long long)seq << 32);
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
    }
};
template <>
struct RingWord<double> {
    static constexpr int n = 2;
    unsigned long long lo, hi;
    __device__ __forceinline__ void load(const unsigned long long* p) {
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
    }
    __device__ __forceinline__ bool has(unsigned int seq) const {
        return (unsigned int)(lo >> 32) == seq && (unsigned int)(hi >> 32) == seq;
    }
    __device__ __forceinline__ double value() const {
        return __hiloint2double((int)(unsigned int)hi, (int)(unsigned int)lo);
    }
    static __device__ __forceinline__ void store(unsigned long long* p, double v, unsigned int seq) {
        const unsigned long long s = (unsigned long long)seq << 32;
        const unsigned long long lo = (unsigned int)__double2loint(v) | s, hi = (unsigned int)__double2hiint(v) | s;
        asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(lo), "l"(hi) : "memory");
    }
};

// Waits until the counter's low half reaches target; false when it gives up.
__device__ __forceinline__ bool count_wait(const unsigned long long* c, unsigned int target, int* err,
                                           unsigned long long* out) {
    unsigned int polls = 0;
    unsigned long long w;
    while ((int)((unsigned int)(w = ld_relaxed(c)) - target) < 0) {
        if ((++polls & 1023u) == 0u) {
            if (vload(err) != 0) return false;
            if (polls > kRingPolls) {
                atomicExch(err, 1);
                return false;
            }
        }
    }
    *out = w;
    return true;
}

// A ring wait that has polled long: gives up (true) when another CTA did or its
// own limit is reached, and tells the others.
static __device__ __noinline__ bool ring_lost(ResSync* s, unsigned int polls) {
    if (vload(&s->bar.err) == 0 && polls < kRingPolls) return false;
    atomicExch(&s->bar.err, 1);
    return true;
}

}  // namespace ntcfd
