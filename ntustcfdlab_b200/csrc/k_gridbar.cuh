// k_gridbar.cuh -- a grid-wide barrier for cooperative launches (every CTA
// co-resident), used by the kernels that run a whole pressure solve.  Every wait is bounded: a barrier
// that gives up sets a shared error flag, so that the other CTAs leave at their next wait.
#pragma once

#include "k_atomics.cuh"

namespace ntcfd {

struct GridBar {
    // one word per parity of the barrier's number.  Low 32 bits: arrivals of the launch; high
    // 32 bits: the sum of the flags added with them (zeroed before a launch)
    unsigned long long word[2];
    int err;
    int pad;
};

// A thread's place in the barriers of a launch: their number so far, and the flags summed by
// each word when it was last read.
struct GridPlace {
    unsigned int n = 0u, seen0 = 0u, seen1 = 0u;
};

constexpr unsigned int kBarrierPolls = 20000000u;   // ~1-2 s of polling without sleep

// Grid-wide barrier of one cooperative launch, split into arrive and wait so
// that a CTA can work between the two.  Barrier n uses the word of n's parity, whose
// low half counts arrivals: each CTA adds 1 with a release
// reduction (after a CTA barrier, so the CTA's earlier global writes are
// published) and does not wait for the add to come back; the m-th barrier of a
// word is passed once its low half reaches m * nblocks.  A CTA may add
// flags to the high half with its arrival (flags << 32), and a waiter reads
// their sum as it sees the barrier pass.  That sum holds this barrier's flags and no later
// ones: a CTA that is past barrier n may arrive at n + 1 before a late waiter reads n, but that is
// the other word, and nobody arrives at n + 2 before the late waiter, having read, arrives at n + 1.
// Waiting polls the word with acquire loads, checks the shared error flag every 1024
// polls and gives up after kBarrierPolls polls, setting the flag so that every
// CTA leaves at its next wait.  Returns false on failure.
__device__ __forceinline__ void grid_arrive(GridBar* b, GridPlace& at, unsigned int flags = 0u) {
    __syncthreads();
    ++at.n;
    if (threadIdx.x == 0) red_add_release(&b->word[at.n & 1u], 1ull | ((unsigned long long)flags << 32));
}

// With over non-null, thread 0 also stores the sum of this barrier's flags to *over before
// the closing CTA barrier, so every thread sees it.
__device__ __forceinline__ bool grid_wait(GridBar* b, GridPlace& at, unsigned int nblocks, int* s_flag,
                                          unsigned int* over = nullptr) {
    if (threadIdx.x == 0) {
        const unsigned int target = ((at.n + 1u) >> 1) * nblocks;
        int fail = 0;
        unsigned int polls = 0;
        unsigned long long w;
        while ((int)((unsigned int)(w = ld_acquire(&b->word[at.n & 1u])) - target) < 0) {
            if ((++polls & 1023u) == 0u) {
                if (vload(&b->err) != 0) { fail = 1; break; }
                if (polls > kBarrierPolls) {
                    atomicExch(&b->err, 1);
                    fail = 1;
                    break;
                }
            }
        }
        *s_flag = fail;
        const unsigned int sum = (unsigned int)(w >> 32), before = at.n & 1u ? at.seen1 : at.seen0;
        if (at.n & 1u) at.seen1 = sum;
        else at.seen0 = sum;
        if (over) *over = sum - before;
    }
    __syncthreads();
    return *s_flag == 0;
}

__device__ __forceinline__ bool grid_sync(GridBar* b, GridPlace& at, unsigned int nblocks, int* s_flag,
                                          unsigned int flags = 0u, unsigned int* over = nullptr) {
    grid_arrive(b, at, flags);
    return grid_wait(b, at, nblocks, s_flag, over);
}

}  // namespace ntcfd
