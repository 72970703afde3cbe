"""CPU: the grid barrier's flags (k_gridbar.cuh, compiled for the host with one
thread per CTA) when one CTA looks late: the others have passed the barrier and
arrived at the next one, as far as the barrier lets them, before it reads.  The
flags that every CTA reads must be those of the barrier it waits at."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

ATOMICS = r"""
#pragma once
#define __device__
#define __forceinline__ inline
struct Index { unsigned int x; };
static const Index threadIdx{0};
inline void __syncthreads() {}
inline int atomicExch(int* p, int v) { return __atomic_exchange_n(p, v, __ATOMIC_SEQ_CST); }
constexpr int kCtas = 4;
constexpr unsigned int kBarriers = 64;
extern thread_local int cta;
extern unsigned int arrived[kCtas];
extern int late;
extern bool stuck;
namespace ntcfd {
inline void red_add_release(unsigned long long* p, unsigned long long v) {
    __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST);
    __atomic_fetch_add(&arrived[cta], 1u, __ATOMIC_SEQ_CST);
}
// The late CTA reads when every other one has arrived at the barrier after this one.
inline unsigned long long ld_acquire(const unsigned long long* p) {
    if (cta == late) {
        const unsigned int n = arrived[cta] < kBarriers ? arrived[cta] + 1 : kBarriers;
        const time_t t0 = time(nullptr);
        for (int c = 0; c < kCtas; ++c)
            while (c != cta && __atomic_load_n(&arrived[c], __ATOMIC_SEQ_CST) < n) {
                std::this_thread::yield();
                if (time(nullptr) - t0 > 20) { stuck = true; break; }
            }
    }
    std::this_thread::yield();
    return __atomic_load_n(p, __ATOMIC_SEQ_CST);
}
inline int vload(const int* p) { return __atomic_load_n(p, __ATOMIC_SEQ_CST); }
}
"""

MAIN = r"""
#include <cstdio>
#include <ctime>
#include <thread>
#include <vector>
#include "k_gridbar.cuh"
thread_local int cta;
unsigned int arrived[kCtas];
int late;
bool stuck;
unsigned int flags_of(int c, unsigned int n) { return (n * 2654435761u >> (c + 7)) % 3u * (n % 5u == 0u ? 1u << 20 : 1u); }
int main() {
    int bad = 0;
    for (late = 0; late < kCtas; ++late) {
        ntcfd::GridBar bar{};
        for (unsigned int& a : arrived) a = 0u;
        std::vector<std::thread> all;
        for (int c = 0; c < kCtas; ++c)
            all.emplace_back([&bar, &bad, c] {
                cta = c;
                ntcfd::GridPlace at;
                for (unsigned int n = 1; n <= kBarriers; ++n) {
                    int failed = 0;
                    unsigned int over = 0u, want = 0u;
                    for (int o = 0; o < kCtas; ++o) want += flags_of(o, n);
                    const bool ok = ntcfd::grid_sync(&bar, at, kCtas, &failed, flags_of(c, n), &over);
                    if (!ok || over != want) __atomic_fetch_add(&bad, 1, __ATOMIC_SEQ_CST);
                }
            });
        for (std::thread& t : all) t.join();
    }
    printf("%d wrong of %u%s\n", bad, kCtas * kCtas * kBarriers, stuck ? ", stuck" : "");
    return bad || stuck ? 1 : 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_flags_belong_to_their_barrier(tmp_path):
    shutil.copy(os.path.join(ROOT, "ntustcfdlab_b200", "csrc", "k_gridbar.cuh"), tmp_path)
    (tmp_path / "k_atomics.cuh").write_text(ATOMICS)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "barrier"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-o", str(exe), str(tmp_path / "main.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
