// k_march.cuh -- a whole pressure solve in one persistent cooperative kernel for
// grids whose correction e does not fit the chip: every sweep marches through
// the planes and updates both colours on the way.
//
// Each CTA owns a tile of rows j and a range of planes k.  A thread owns the cell
// pairs x (i = 2x-1 odd and i = 2x even, one red and one black) of RJ rows and
// walks k: at step k it updates the red cells of plane k and, one plane behind,
// the black cells of plane k-1, whose red neighbours k-2, k-1, k it has just made.
// The neighbours along k are the thread's own registers, those along j and in
// the next pair come from shared memory.  A copying warp brings the tile's rows of the
// planes in by bulk copies, kMarchAhead steps ahead (a plane's rows of a tile lie
// together, one copy each); the updating warps wait for a step's copies and for one
// another's new red cells on shared-memory barriers, which they arrive at before the
// black half of a step, so that half covers the wait.  The black cells of a
// tile need the red cells of one row and plane around it, which the CTA updates
// for itself from the same old values as their owner does (the same bits); the
// sweep goes from one pair of arrays to another, since a neighbour still reads
// the old values.  FP32 updates two rows in one packed instruction.
//
// One grid barrier ends a sweep and carries the stop test's verdicts (GS.f90:11,
// 53); the restarts of the defect correction and the last p += e run in the
// kernel too.  Every wait is bounded; one that gives up ends the solve with an error.
//
// Bound: per cell and sweep e is read and written once and d read once, 12 bytes FP32,
// 24 FP64, against 16 and 40 of two half-sweep passes (which also read 1/diag in FP64;
// here it is formed from the 1-D tables).  128x256x384: FP64 57.5 us a sweep (5.25 TB/s of
// those bytes; 119.8 before, by half-sweeps), FP32 35.9 us (58.7 before), where
// the chain of a step (copies in, shared loads, two dependent updates, barrier: 0.5 to 0.8 us)
// bounds it, with 38% of the issue slots used; a restart 92 us (85).  64x192x256: FP64 19.7 (50.1),
// FP32 11.3 and its restart 21 us (39).
// What was tried: 2, 6 and 8 rows a thread (FP32 8 rows and 256 threads: 102 us, too
// few warps; FP64 2 rows and 512: 65 us), copies 3 steps ahead (the same time), per-thread asynchronous
// copies and one CTA barrier a step (FP64 81 us), loads into registers a step ahead
// (FP64 124 us).
#pragma once

#include <type_traits>

#include "k_exchange.cuh"
#include "k_sor_math.cuh"
#include "ntcfd_common.cuh"

namespace ntcfd {

// Launch plan and layout.  The colour arrays hold, per plane k = -1..nz+2 and row
// j = -1.. (ny + 4 + 2 RJ of them), HP pairs: x = 1..H at element x - 1, the rest 0 (so that
// x - 1 and x + 1 beyond a row read 0), after kMarchPad elements of 0.  The ghost rows
// and planes are 0 and never written, so the sweep loads without bounds checks.
struct MarchPlan {
    int H = 0, HP = 0;       // pairs per row, and the row pitch
    int groups = 0;          // row groups of a CTA (RJ rows each); H * groups threads update, rounded up to a warp
    int nbj = 0, nbk = 0;    // tiles along j, ranges along k (balanced)
    int nt = 0;              // threads: those, and the copying warp
    size_t smem = 0;
    size_t elems = 0;        // of one colour array
};
constexpr int kMarchPad = 8;
// Row pitches with an instance of their own (the pitch as a constant makes every row
// of a thread a constant offset: 25% fewer instructions); a grid takes the first that
// holds its H pairs and a 0.
constexpr int kMarchHP[] = {24, 40, 72, 120};
constexpr int kMarchRJ = 4, kMarchNT = 352;                     // rows of a thread, updating threads of a CTA at most
constexpr int kMarchAhead = 2;                                  // steps a copy runs ahead of its use
constexpr int kMarchPlanes = (kMarchAhead + 2) + 3 * (kMarchAhead + 1) + 2;   // shared planes of a tile
__host__ __device__ constexpr int march_pad(int HP) { return HP + 8; }        // words before and after them

template <class Tc>
struct MarchArgs {
    Geom g;
    SorCoef<Tc> sc;
    int H, HP, groups, nbj, nbk;
    double* p;
    const double* b;
    Tc* f;                   // six colour arrays, `elems` apart: e (two buffers, red and black each), d
    int elems;
    Ctl* ctl;
    ResSync* sync;
    double omega, zeta;
    int itmax, cycle_len, check_every;
};

// The largest |change| of a thread, NaN kept: one instruction per cell in FP32,
// an order-preserving pattern in FP64.
template <class Tc>
struct Change;
template <>
struct Change<float> {
    float m = 0.0f;
    __device__ __forceinline__ void take(float d) { asm("max.NaN.f32 %0, %0, %1;" : "+f"(m) : "f"(fabsf(d))); }
    __device__ __forceinline__ unsigned long long bits() const { return widen_bits(abs_bits(m)); }
};
template <>
struct Change<double> {
    unsigned long long m = 0ull;
    __device__ __forceinline__ void take(double d) {
        const unsigned long long b = abs_bits(d);
        m = b > m ? b : m;
    }
    __device__ __forceinline__ unsigned long long bits() const { return m; }
};

// A CTA's tile and a thread's place in it.
struct MarchTile {
    int ja, jb, ka, kb;      // own rows and planes
    int x, j0;               // the thread's pair (1..H) and first row
    bool act, ok1;           // it has cells; the even one of the pair exists
    int row0, ps;            // its first row in plane 0, and the plane pitch, of a colour array
    int grp;
    template <class Tc>
    __device__ __forceinline__ explicit MarchTile(const MarchArgs<Tc>& a) {
        constexpr int RJ = kMarchRJ;
        const Geom& g = a.g;
        const int bj = blockIdx.x % a.nbj, bk = blockIdx.x / a.nbj, tid = threadIdx.x;
        ja = 1 + brick_start(bj, g.ny, a.nbj);
        jb = brick_start(bj + 1, g.ny, a.nbj);
        ka = 1 + brick_start(bk, g.nz, a.nbk);
        kb = brick_start(bk + 1, g.nz, a.nbk);
        grp = min(tid / a.H, a.groups - 1);
        const int xt = tid - grp * a.H + 1;           // beyond H: a thread without cells
        act = xt <= a.H;
        x = min(xt, a.H);
        j0 = ja - 2 + grp * RJ;
        ok1 = 2 * x <= g.nx;
        ps = (g.ny + 4 + 2 * RJ) * a.HP;
        row0 = kMarchPad + (j0 + 1) * a.HP + x - 1 + ps;
    }
};

// The first defect of a solve: the FP64 defect of p (defect_value) of the own cells.
// Rows outside the tile repeat one inside, so that every load can be issued at once.
template <class Tc>
__device__ __noinline__ void march_defect(const MarchArgs<Tc>& a) {
    constexpr int RJ = kMarchRJ;
    const Geom& g = a.g;
    const MarchTile m(a);
    if (!m.act) return;
    const double gE[2] = {g.cE[2 * m.x - 1], g.cE[min(2 * m.x, g.nx + 2)]};
    const double gW[2] = {g.cW[2 * m.x - 1], g.cW[min(2 * m.x, g.nx + 2)]};
    for (int k = m.ka; k <= m.kb; ++k) {
        const double fF = g.cF[k], fB = g.cB[k];
#pragma unroll
        for (int r = 0; r < RJ; ++r) {
            const int j = min(max(m.j0 + r, m.ja), m.jb);
            const double nN = g.cN[j], nS = g.cS[j];
            const long long c = nat(g, 2 * m.x - 1, j, k);
            const double* pp = a.p + c;
            const double v[4] = {pp[-1], pp[0], pp[1], pp[2]};
            const double b[2] = {a.b[c], a.b[c + 1]};
            Tc* const d = a.f + 4 * a.elems + m.row0 + (j - m.j0) * a.HP + k * m.ps;
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const double rd = rcp_rn(((gE[t] + gW[t]) + (nN + nS)) + (fF + fB));
                const double dv = defect_value(gE[t], v[t + 2], gW[t], v[t], nN, pp[t + g.px], nS, pp[t - g.px], fF,
                                               pp[t + g.pz], fB, pp[t - g.pz], rd, b[t], v[t + 1]);
                if (j == m.j0 + r && (t == 0 || m.ok1)) d[((t + 1 + j + k) & 1) * a.elems] = (Tc)dv;
            }
        }
    }
}

// p += e (buffer cur) of the own cells.
template <class Tc>
__device__ __noinline__ void march_correct(const MarchArgs<Tc>& a, int cur) {
    constexpr int RJ = kMarchRJ;
    const Geom& g = a.g;
    const MarchTile m(a);
    if (!m.act) return;
    const Tc *const R = a.f + 2 * cur * a.elems, *const B = R + a.elems;
#pragma unroll 2
    for (int k = m.ka; k <= m.kb; ++k) {
        Tc er[RJ], eb[RJ];
        double2 pv[RJ];
        bool own[RJ];
#pragma unroll
        for (int r = 0; r < RJ; ++r) {
            const int j = m.j0 + r, c = m.row0 + r * a.HP + k * m.ps;
            own[r] = j >= m.ja && j <= m.jb;
            if (!own[r]) continue;
            er[r] = __ldcg(R + c);
            eb[r] = __ldcg(B + c);
            pv[r] = *reinterpret_cast<const double2*>(a.p + nat(g, 2 * m.x - 1, j, k));
        }
#pragma unroll
        for (int r = 0; r < RJ; ++r) {
            if (!own[r]) continue;
            const int j = m.j0 + r;
            const bool odd = (j + k) & 1;             // the pair's odd cell is the red one
            double* const pp = a.p + nat(g, 2 * m.x - 1, j, k);
            const double v0 = pv[r].x + (double)(odd ? er[r] : eb[r]), v1 = pv[r].y + (double)(odd ? eb[r] : er[r]);
            if (m.ok1) *reinterpret_cast<double2*>(pp) = make_double2(v0, v1);
            else *pp = v0;
        }
    }
}

// The values of W rows of a thread in one operand: two in FP32 (packed arithmetic: one
// instruction for both, each rounded as alone), one in FP64.  A sweep holds its
// coefficients negated in FP32 (the packed operations have no sign of their own).
template <class Tc>
struct Rows;
template <>
struct Rows<float> {
    static constexpr int W = 2;
    unsigned long long v;
    static __device__ __forceinline__ Rows of(float a, float b) {
        Rows r;
        asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
        return r;
    }
    __device__ __forceinline__ float get(int q) const {
        float a, b;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
        return q ? b : a;
    }
    static __device__ __forceinline__ float sign(float c) { return -c; }
};
__device__ __forceinline__ Rows<float> mul_rn(Rows<float> a, Rows<float> b) {
    Rows<float> r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ Rows<float> fma_rn(Rows<float> a, Rows<float> b, Rows<float> c) {
    Rows<float> r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ Rows<float> add_rn(Rows<float> a, Rows<float> b) {
    Rows<float> r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ Rows<float> sub_rn(Rows<float> a, Rows<float> b) {
    Rows<float> r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
template <>
struct Rows<double> {
    static constexpr int W = 1;
    double v;
    static __device__ __forceinline__ Rows of(double a, double) { return {a}; }
    __device__ __forceinline__ double get(int) const { return v; }
    static __device__ __forceinline__ double sign(double c) { return c; }
};
__device__ __forceinline__ Rows<double> mul_rn(Rows<double> a, Rows<double> b) { return {mul_rn(a.v, b.v)}; }
__device__ __forceinline__ Rows<double> fma_rn(Rows<double> a, Rows<double> b, Rows<double> c) {
    return {fma_rn(a.v, b.v, c.v)};
}
__device__ __forceinline__ Rows<double> add_rn(Rows<double> a, Rows<double> b) { return {a.v + b.v}; }
__device__ __forceinline__ Rows<double> sub_rn(Rows<double> a, Rows<double> b) { return {sub_rn(a.v, b.v)}; }

// 1 / diag of the coefficient sum s, with the coefficients' sign (rdiag_near, two rows at once).
__device__ __forceinline__ Rows<float> march_rd(Rows<float> s) {
    float a, b;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(-s.get(0)));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(-s.get(1)));
    const Rows<float> x = Rows<float>::of(a, b);
    return fma_rn(x, fma_rn(s, x, Rows<float>::of(1.0f, 1.0f)), x);
}
__device__ __forceinline__ Rows<double> march_rd(Rows<double> s) { return {rdiag_near(s.v)}; }

// Barriers in shared memory (mbarrier) and the bulk copies that complete on them.
__device__ __forceinline__ unsigned int sm32(const void* p) { return (unsigned int)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* b, unsigned int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sm32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(sm32(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long* b, unsigned int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(sm32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned long long* b, unsigned int parity) {
    unsigned int ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n"
                 " selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(sm32(b)), "r"(parity)
                 : "memory");
    return ok != 0u;
}
constexpr long long kMarchClocks = 1ll << 32;    // of waiting at a shared barrier before giving up (2 s)
// Waits for the phase of a parity; false when it gives up.
__device__ __forceinline__ bool mbar_wait(unsigned long long* b, unsigned int parity) {
    if (mbar_try(b, parity)) return true;
    const long long t0 = clock64();
#pragma unroll 1
    while (clock64() - t0 < kMarchClocks)
        if (mbar_try(b, parity)) return true;
    return false;
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, unsigned int bytes, unsigned long long* b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sm32(dst)),
                 "l"(src), "r"(bytes), "r"(sm32(b))
                 : "memory");
}
// Orders this thread's (and, after a barrier, the CTA's) plain accesses with bulk copies.
__device__ __forceinline__ void fence_bulk() { asm volatile("fence.proxy.async;" ::: "memory"); }

struct MarchBars {
    unsigned long long full[kMarchAhead + 1];    // a step's copies have arrived
    unsigned long long done[kMarchAhead + 1];    // every warp has read a step's planes and written its new red
};

// Place of a step in the barriers' rings: slot and phase.
struct MarchPos {
    int slot;
    unsigned int lap;
    __device__ __forceinline__ explicit MarchPos(unsigned long long n)
        : slot((int)(n % (kMarchAhead + 1))), lap((unsigned int)(n / (kMarchAhead + 1)) & 1u) {}
    __device__ __forceinline__ void next() {
        if (++slot == kMarchAhead + 1) {
            slot = 0;
            lap ^= 1u;
        }
    }
    // the step before
    __device__ __forceinline__ MarchPos prev() const {
        MarchPos p = *this;
        p.slot = slot ? slot - 1 : kMarchAhead;
        p.lap = slot ? lap : lap ^ 1u;
        return p;
    }
};

// The copying thread's end of a march of `issued` steps, the last of them before pos: it waits
// (with the limit of every wait) until its last copies have landed, also where the march was
// given up, so that no copy is in flight when the CTA leaves.  In a march that ran through, the
// updating warps have waited for the same copies.
__device__ __forceinline__ bool march_drain(MarchBars* bars, MarchPos pos, int issued) {
    bool ok = true;
    for (int q = min(issued, kMarchAhead + 1); q > 0; --q) {
        pos = pos.prev();
        ok = mbar_wait(bars->full + pos.slot, pos.lap) && ok;
    }
    return ok;
}

// The restart of a correction cycle: p += e (buffer cur) and d = the FP64 defect of
// p + e (defect_update), in a march with the sweep's copies: e of plane k+1 and d
// of plane k.
template <class Tc, int HP>
__device__ __noinline__ void march_restart(const MarchArgs<Tc>& a, MarchBars* bars, int cur, unsigned long long n0,
                                           bool* lost) {
    constexpr int RJ = kMarchRJ, D = kMarchAhead;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Geom& g = a.g;
    const MarchTile m(a);
    const int ka = m.ka, kb = m.kb, ps = m.ps, tid = threadIdx.x, nt = blockDim.x - 32;
    // shared planes: red and black e (D + 2 each, in turn), {red d, black d} (D + 1)
    const int PL = a.groups * RJ * HP;
    Tc* const SE = reinterpret_cast<Tc*>(smem_raw) + march_pad(HP);
    Tc* const SD = SE + 2 * (D + 2) * PL;
    const int me = m.grp * RJ * HP + m.x - 1;
    const double gE[2] = {g.cE[2 * m.x - 1], g.cE[min(2 * m.x, g.nx + 2)]};
    const double gW[2] = {g.cW[2 * m.x - 1], g.cW[min(2 * m.x, g.nx + 2)]};
    bool own[RJ];
#pragma unroll
    for (int r = 0; r < RJ; ++r) own[r] = m.act && m.j0 + r >= m.ja && m.j0 + r <= m.jb;
    const int tile0 = kMarchPad + (m.ja - 1) * HP + ps;   // the tile's first row (ja - 2), plane 0
    const int Ri = 2 * cur * a.elems, Bi = Ri + a.elems, Di = 4 * a.elems;
    Tc* const f = a.f;
    auto wrap = [&](int s, int n) { return s + 1 == n ? 0 : s + 1; };
    MarchPos pos(n0);
    if (tid >= nt) {                                  // the copying warp
        bool ok = true;
        if (tid == nt) {
            constexpr unsigned int w = sizeof(Tc);
            int ef = 1, issued = 0;
            fence_bulk();
            for (int k = ka; k <= kb; ++k, ++issued) {
                if (k > ka + D) ok = mbar_wait(bars->done + pos.slot, pos.lap ^ 1u);
                if (!ok) break;
                const int sR = Ri + tile0 + k * ps, sB = sR + a.elems, sd = Di + tile0 + k * ps;
                Tc *const e = SE + 2 * ef * PL, *const d = SD + 2 * pos.slot * PL;
                unsigned long long* const bar = bars->full + pos.slot;
                mbar_expect(bar, (k == ka ? 6u : 4u) * w * PL);
                if (k == ka) {
                    bulk_copy(SE, f + sR, w * PL, bar);
                    bulk_copy(SE + PL, f + sB, w * PL, bar);
                }
                bulk_copy(e, f + (sR + ps), w * PL, bar);
                bulk_copy(e + PL, f + (sB + ps), w * PL, bar);
                bulk_copy(d, f + sd, w * PL, bar);
                bulk_copy(d + PL, f + (sd + a.elems), w * PL, bar);
                ef = wrap(ef, D + 2);
                pos.next();
            }
            if (!march_drain(bars, pos, issued) || !ok) *lost = true;
        }
        return;
    }
    int es = 0;                                       // place of e of plane k
    Tc Rm[RJ], Bm[RJ];                                // e of plane k-1
    int at = m.row0 + ka * ps;
#pragma unroll
    for (int r = 0; r < RJ; ++r) {
        Rm[r] = __ldcg(f + (Ri + at - ps) + r * HP);
        Bm[r] = __ldcg(f + (Bi + at - ps) + r * HP);
    }
    bool ok = true;
    auto step = [&](auto qq, int k) __attribute__((always_inline)) {
        constexpr int Q = decltype(qq)::value;        // parity of j0 + k
        double2 pv[RJ];
        double* const pp = a.p + nat(g, 2 * m.x - 1, m.j0, k);
#pragma unroll
        for (int r = 0; r < RJ; ++r)
            if (own[r]) pv[r] = *reinterpret_cast<const double2*>(pp + r * g.px);
        ok = mbar_wait(bars->full + pos.slot, pos.lap);
        const int en = wrap(es, D + 2);
        const Tc *const sR = SE + 2 * es * PL + me, *const sB = sR + PL;
        const Tc *const sRn = SE + 2 * en * PL + me, *const sBn = sRn + PL;
        const Tc* const sd = SD + 2 * pos.slot * PL + me;
        Tc R0[RJ + 2], B0[RJ + 2], ewr[RJ], ewb[RJ], Rp[RJ], Bp[RJ], dr[RJ], db[RJ];   // ew: the outer neighbour of red, of black
#pragma unroll
        for (int r = 0; r < RJ + 2; ++r) {
            R0[r] = sR[(r - 1) * HP];
            B0[r] = sB[(r - 1) * HP];
        }
#pragma unroll
        for (int r = 0; r < RJ; ++r) {
            const int o = r * HP, h = (1 ^ Q ^ (r & 1)) ? 1 : -1;
            ewr[r] = sB[o + h];
            ewb[r] = sR[o - h];
            Rp[r] = sRn[o];
            Bp[r] = sBn[o];
            dr[r] = sd[o];
            db[r] = sd[PL + o];
        }
        ok = __all_sync(0xffffffffu, ok);
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(bars->done + pos.slot);
        const double fF = g.cF[k], fB = g.cB[k];
        Tc* const dp = f + (Di + at);
#pragma unroll
        for (int r = 0; r < RJ; ++r) {
            const int tr = 1 ^ Q ^ (r & 1);           // the red cell of the pair is the even one
            const Tc er = R0[r + 1], eb = B0[r + 1];
            if (own[r]) {
                const double nN = g.cN[m.j0 + r], nS = g.cS[m.j0 + r];
                // red; then black, whose neighbours across the pair are the other way round
                const double d0 = defect_update(gE[tr], tr ? ewr[r] : eb, gW[tr], tr ? eb : ewr[r], nN, B0[r + 2], nS, B0[r],
                                                fF, Bp[r], fB, Bm[r], dr[r], er);
                const double d1 = defect_update(gE[1 - tr], tr ? er : ewb[r], gW[1 - tr], tr ? ewb[r] : er, nN, R0[r + 2], nS,
                                                R0[r], fF, Rp[r], fB, Rm[r], db[r], eb);
                if (m.ok1 || tr == 0) dp[r * HP] = (Tc)d0;
                if (m.ok1 || tr == 1) dp[a.elems + r * HP] = (Tc)d1;
                const double v0 = pv[r].x + (double)(tr ? eb : er), v1 = pv[r].y + (double)(tr ? er : eb);
                if (m.ok1) *reinterpret_cast<double2*>(pp + r * g.px) = make_double2(v0, v1);
                else pp[r * g.px] = v0;
            }
            Rm[r] = er;
            Bm[r] = eb;
        }
        at += ps;
        es = en;
        pos.next();
    };
#pragma unroll 1
    for (int k = ka; k <= kb; ++k) {
        if ((m.j0 + k) & 1) step(std::integral_constant<int, 1>{}, k);
        else step(std::integral_constant<int, 0>{}, k);
        if (!ok) break;
    }
    fence_bulk();                                     // the new d
    if (!ok) *lost = true;
}

// One sweep from buffer `cur` (first: e is 0) into the other; the thread's max
// |change|.  The tile's rows of a plane lie together in each colour array and are
// copied to shared memory kAhead steps before their step: old black of plane k+1,
// old red and red d of plane k, black d of plane k-1.
template <class Tc, int HP>
__device__ __noinline__ unsigned long long march_sweep(const MarchArgs<Tc>& a, MarchBars* bars, int cur, bool first,
                                                       unsigned long long n0, bool* lost) {
    constexpr int RJ = kMarchRJ, D = kMarchAhead;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Geom& g = a.g;
    const MarchTile m(a);
    const int ka = m.ka, kb = m.kb, ps = m.ps, tid = threadIdx.x, nt = blockDim.x - 32;
    const bool act = m.act;
    // shared planes of the tile's rows (pitch HP): old black (D + 2), {old red, red d, black d}
    // (D + 1), new red (2); a row and more before and after, where the rows outside a tile's
    // first and last are read (their cells are never used)
    const int PL = a.groups * RJ * HP;
    Tc* const SB = reinterpret_cast<Tc*>(smem_raw) + march_pad(HP);
    Tc* const SO = SB + (D + 2) * PL;
    Tc* const SR = SO + 3 * (D + 1) * PL;
    const Tc* const cFB = SR + 2 * PL + march_pad(HP);   // cF, cB of planes ka-1 ..
    const int me = m.grp * RJ * HP + m.x - 1;
    using V = Rows<Tc>;
    constexpr int W = V::W, RV = RJ / W;              // operands of a thread: rows v, v + RV
    static_assert(RV % 2 == 0, "the rows of an operand have one parity");
    auto both = [](Tc c) { return V::of(c, c); };
    const V om = both((Tc)a.omega);
    // Coefficients.  A cell outside the domain keeps e = 0 without any test: its own plane,
    // row or pair holds zeros, and the coefficient of its one neighbour inside is 0 here.
    const Tc e2[2] = {a.sc.cE[2 * m.x - 1], m.ok1 ? a.sc.cE[2 * m.x] : Tc(1)};
    const Tc w2[2] = {a.sc.cW[2 * m.x - 1], m.ok1 ? a.sc.cW[2 * m.x] : Tc(0)};
    const V cE[2] = {both(V::sign(e2[0])), both(V::sign(e2[1]))}, cW[2] = {both(V::sign(w2[0])), both(V::sign(w2[1]))};
    V cN[RV], cS[RV], sENS[2][RV];                    // sENS: the i and j part of a cell's diagonal
    bool own[RJ];                                     // the row belongs to this tile
    {
        Tc n[RJ], s[RJ];
#pragma unroll
        for (int r = 0; r < RJ; ++r) {
            const int j = m.j0 + r;
            const bool in = j >= 1 && j <= g.ny;
            own[r] = act && j >= m.ja && j <= m.jb;
            n[r] = in ? a.sc.cN[j] : Tc(0);
            s[r] = in ? a.sc.cS[j] : Tc(0);
        }
#pragma unroll
        for (int v = 0; v < RV; ++v) {
            const int u = W > 1 ? v + RV : v;
            cN[v] = V::of(V::sign(n[v]), V::sign(n[u]));
            cS[v] = V::of(V::sign(s[v]), V::sign(s[u]));
#pragma unroll
            for (int t = 0; t < 2; ++t)
                sENS[t][v] = V::of((e2[t] + w2[t]) + (n[v] + s[v]), (e2[t] + w2[t]) + (n[u] + s[u]));
        }
    }
    Tc* const f = a.f;
    const int elems = a.elems;
    const int Ri = 2 * cur * elems, Bi = Ri + elems, Ro = 2 * (cur ^ 1) * elems, Bo = Ro + elems;
    const int tile0 = kMarchPad + (m.ja - 1) * HP + ps;   // the tile's first row (ja - 2), plane 0
    auto wrap = [&](int s, int n) { return s + 1 == n ? 0 : s + 1; };
    MarchPos pos(n0);
    if (tid >= nt) {                                  // the copying warp
        bool ok = true;
        if (tid == nt) {
            // step k's copies; a cycle's first sweep copies a plane of zeros (k = -1) for e
            constexpr unsigned int w = sizeof(Tc);
            int bf = 1, issued = 0;
            fence_bulk();
            for (int k = ka - 1; k <= kb + 1; ++k, ++issued) {
                if (k > ka - 1 + D) ok = mbar_wait(bars->done + pos.slot, pos.lap ^ 1u);
                if (!ok) break;
                const int sB = Bi + tile0 + (first ? -1 : k + 1) * ps, sR = Ri + tile0 + (first ? -1 : k) * ps;
                const int sd = 4 * elems + tile0 + k * ps;
                Tc* const o = SO + 3 * pos.slot * PL;
                unsigned long long* const bar = bars->full + pos.slot;
                mbar_expect(bar, (k < ka ? 5u : 4u) * w * PL);
                if (k < ka) bulk_copy(SB, f + (Bi + tile0 + (first ? -1 : k) * ps), w * PL, bar);
                bulk_copy(SB + bf * PL, f + sB, w * PL, bar);
                bulk_copy(o, f + sR, w * PL, bar);
                bulk_copy(o + PL, f + sd, w * PL, bar);
                bulk_copy(o + 2 * PL, f + (sd + (elems - ps)), w * PL, bar);
                bf = wrap(bf, D + 2);
                pos.next();
            }
            if (!march_drain(bars, pos, issued) || !ok) *lost = true;
        }
        return 0ull;
    }
    MarchPos before = pos.prev();
    int bs = 0;                                       // place of black of plane k
    V Bm[RV], B0[RV], R1[RV], R2[RV];                // own old black of planes k-1, k, new red of k-1, k-2
    int at = m.row0 + (ka - 1) * ps;                  // the thread's first row in plane k
#pragma unroll
    for (int v = 0; v < RV; ++v) {
        auto ld = [&](int off, int r) { return first ? Tc(0) : __ldcg(f + (Bi + at + off) + r * HP); };
        Bm[v] = V::of(ld(-ps, v), ld(-ps, v + RV * (W - 1)));
        B0[v] = V::of(ld(0, v), ld(0, v + RV * (W - 1)));
        R1[v] = R2[v] = both(Tc(0));
    }
    V cF1 = both(Tc(0)), cB1 = cF1, sFB1 = cF1;       // of plane k-1
    // the neighbours along j of operand v: its own rows' X, `up` and `dn` from shared memory
    auto north = [&](const V* X, int v, Tc up) __attribute__((always_inline)) {
        return v + 1 < RV ? X[v + 1 < RV ? v + 1 : 0] : V::of(W > 1 ? X[0].get(1) : up, up);
    };
    auto south = [&](const V* X, int v, Tc dn) __attribute__((always_inline)) {
        return v > 0 ? X[v > 0 ? v - 1 : 0] : V::of(dn, X[RV - 1].get(0));
    };
    Change<Tc> ch;
    auto step = [&](auto qq, int k) __attribute__((always_inline)) {
        constexpr int Q = decltype(qq)::value;        // parity of j0 + k
        bool ok = mbar_wait(bars->full + pos.slot, pos.lap);         // step k's copies are in
        ok = mbar_wait(bars->done + before.slot, before.lap) && ok;  // step k-1 is done everywhere
        const bool more = k <= kb;
        const Tc f1 = cFB[2 * (k - ka + 1)], b1 = cFB[2 * (k - ka + 1) + 1];
        const V cF = both(V::sign(f1)), cB = both(V::sign(b1)), sFB = both(f1 + b1);
        const int bn = wrap(bs, D + 2);
        const Tc* const sb = SB + bs * PL + me;       // black of plane k
        const Tc* const sbn = SB + bn * PL + me;      // black of plane k+1
        const Tc* const so = SO + 3 * pos.slot * PL + me;   // old red and red d of plane k, black d of k-1
        Tc* const srn = SR + (k & 1) * PL + me;       // new red of plane k
        const Tc* const sr = SR + ((k + 1) & 1) * PL + me;   // and of k-1
        V ewb[RV], ewr[RV], Bp[RV], Rc[RV], dr[RV], db[RV], Rk[RV];
        const Tc nb = sb[RJ * HP], sbv = sb[-HP], nr = sr[RJ * HP], srv = sr[-HP];
#pragma unroll
        for (int v = 0; v < RV; ++v) {
            const int o = v * HP, u = o + (W - 1) * RV * HP, h = (1 ^ Q ^ (v & 1)) ? 1 : -1;
            ewb[v] = V::of(sb[o + h], sb[u + h]);
            Bp[v] = V::of(sbn[o], sbn[u]);
            Rc[v] = V::of(so[o], so[u]);
            dr[v] = V::of(so[PL + o], so[PL + u]);
            ewr[v] = V::of(sr[o + h], sr[u + h]);
            db[v] = V::of(so[2 * PL + o], so[2 * PL + u]);
        }
        Tc* const fr = f + (Ro + at);                 // new red of plane k, new black of k-1
        Tc* const fb = f + (Bo + at - ps);
        // red cells of plane k
        const bool st = k >= ka && more;
#pragma unroll
        for (int v = 0; v < RV; ++v) {
            const int t = 1 ^ Q ^ (v & 1);
            const V ew = ewb[v], ctr = B0[v], rd = march_rd(add_rn(sENS[t][v], sFB));
            const V diff = sor_update(cE[t], t ? ew : ctr, cW[t], t ? ctr : ew, cN[v], north(B0, v, nb), cS[v],
                                      south(B0, v, sbv), cF, Bp[v], cB, Bm[v], rd, dr[v], Rc[v], om, &Rk[v]);
#pragma unroll
            for (int q = 0; q < W; ++q) {
                const int r = v + q * RV;
                if (st && own[r]) {
                    ch.take(diff.get(q));
                    fr[r * HP] = Rk[v].get(q);
                }
                if (act) srn[r * HP] = Rk[v].get(q);
            }
        }
        ok = __all_sync(0xffffffffu, ok);             // a warp leaves together
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(bars->done + pos.slot);   // the black cells need nothing more of the planes
        // black cells of plane k-1
        if (k > ka) {
#pragma unroll
            for (int v = 0; v < RV; ++v) {
                const int t = 1 ^ Q ^ (v & 1);
                const V ew = ewr[v], ctr = R1[v], rd = march_rd(add_rn(sENS[t][v], sFB1));
                V e1;
                const V diff = sor_update(cE[t], t ? ew : ctr, cW[t], t ? ctr : ew, cN[v], north(R1, v, nr), cS[v],
                                          south(R1, v, srv), cF1, Rk[v], cB1, R2[v], rd, db[v], Bm[v], om, &e1);
#pragma unroll
                for (int q = 0; q < W; ++q) {
                    const int r = v + q * RV;
                    if (own[r]) {
                        ch.take(diff.get(q));
                        fb[r * HP] = e1.get(q);
                    }
                }
            }
        }
#pragma unroll
        for (int v = 0; v < RV; ++v) {
            Bm[v] = B0[v];
            B0[v] = Bp[v];
            R2[v] = R1[v];
            R1[v] = Rk[v];
        }
        sFB1 = sFB;
        at += ps;
        cF1 = cF;
        cB1 = cB;
        bs = bn;
        before = pos;
        pos.next();
        return ok;
    };
    bool ok = true;
#pragma unroll 1
    for (int k = ka - 1 - ((m.ja + ka + 1) & 1); k <= kb + 1; k += 2) {   // j0 + k even
        if (k >= ka - 1) ok = step(std::integral_constant<int, 0>{}, k);
        if (k <= kb && ok) ok = step(std::integral_constant<int, 1>{}, k + 1);
        if (!ok) break;
    }
    fence_bulk();                                     // the new e, which the next sweep copies
    if (!ok) *lost = true;
    return ch.bits();
}

template <class Tc, int HP>
__global__ void __launch_bounds__(kMarchNT + 32, 1) k_sor_march(const __grid_constant__ MarchArgs<Tc> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_flag, s_nan[2];
    __shared__ unsigned int s_over;               // CTAs above zeta, 2^20 per one that met a NaN, of a sweep
    __shared__ unsigned long long s_max[kMarchNT / 32 + 1];
    __shared__ MarchBars s_bars;
    __shared__ bool s_lost;
    const int tid = threadIdx.x;
    {
        const int words = kMarchPlanes * a.groups * kMarchRJ * a.HP + 2 * march_pad(a.HP);
        Tc* const sm = reinterpret_cast<Tc*>(smem_raw);
        for (int q = tid; q < words; q += blockDim.x) sm[q] = Tc(0);
        const int bk = blockIdx.x / a.nbj, k1 = brick_start(bk, a.g.nz, a.nbk), nk = brick_start(bk + 1, a.g.nz, a.nbk) - k1 + 2;
        for (int q = tid; q < nk; q += blockDim.x) {   // planes ka-1 .. kb+1, 0 outside the domain
            const int k = k1 + q;
            const bool in = k >= 1 && k <= a.g.nz;
            sm[words + 2 * q] = in ? a.sc.cF[k] : Tc(0);
            sm[words + 2 * q + 1] = in ? a.sc.cB[k] : Tc(0);
        }
    }
    if (tid == 0) {
        s_nan[0] = s_nan[1] = 0;
        s_lost = false;
        for (int q = 0; q <= kMarchAhead; ++q) {
            mbar_init(s_bars.full + q, 1u);
            mbar_init(s_bars.done + q, blockDim.x / 32 - 1);
        }
    }
    march_defect<Tc>(a);
    fence_bulk();
    unsigned int steps;                               // of a sweep
    unsigned long long n = 0ull;                      // steps so far: the phases of the shared barriers
    {
        const int bk = blockIdx.x / a.nbj;
        steps = brick_start(bk + 1, a.g.nz, a.nbk) - brick_start(bk, a.g.nz, a.nbk) + 2;
    }
    GridPlace at;
    const unsigned int nblocks = gridDim.x;
    bool failed = !grid_sync(&a.sync->bar, at, nblocks, &s_flag);

    int done = 0, done_c = 0, cycles = 0, cur = 0;    // cur: the buffer that holds e
    bool conv = false, nonfinite = false, tested = false;
    unsigned long long chs = 0ull;                    // this thread's max |change| of the last sweep

    auto above = [&](unsigned long long b) { return !(__longlong_as_double((long long)b) <= a.zeta); };
    // Whether a wait of this CTA gave up, after a CTA barrier: it then leaves without
    // arriving at the grid barrier, and the error flag takes the others out of it.
    auto lost = [&]() {
        if (s_lost && tid == 0) atomicExch(&a.sync->bar.err, 1);
        return s_lost;
    };

    while (!failed) {
        done_c = 0;
#pragma unroll 1
        for (int s = 0; done + s < a.itmax && s < a.cycle_len; ++s) {
            const int ik = done + s + 1, par = ik & 1;
            const unsigned long long cb = march_sweep<Tc, HP>(a, &s_bars, cur, s == 0, n, &s_lost);
            n += steps;
            cur ^= 1;
            if (cb >= kInfBits) s_nan[par] = 1;
            const int any = __syncthreads_or(above(cb));
            if (lost() || !grid_sync(&a.sync->bar, at, nblocks, &s_flag,
                                     (any ? 1u : 0u) + (tid == 0 && s_nan[par] ? 1u << 20 : 0u), &s_over)) {
                failed = true;
                break;
            }
            const unsigned int over = s_over;
            chs = cb;
            done_c = s + 1;
            // every check_every sweeps of the cycle and at its end, as the half-sweep loops test
            if (a.check_every == 1 || ik >= a.itmax || s + 1 >= a.cycle_len || (s + 1) % a.check_every == 0) {
                tested = true;
                nonfinite = over >= (1u << 20);
                conv = over == 0u;
                if (conv || nonfinite) break;
            }
        }
        done += done_c;
        ++cycles;
        // another cycle only when this one ended on its length
        if (failed || conv || nonfinite || done_c < a.cycle_len || done >= a.itmax) break;
        march_restart<Tc, HP>(a, &s_bars, cur, n, &s_lost);
        n += steps - 2;
        __syncthreads();
        if (lost() || !grid_sync(&a.sync->bar, at, nblocks, &s_flag)) failed = true;
    }
    if (!failed && done > 0) march_correct<Tc>(a, cur);
    double last = 0.0;
    if (!failed && tested) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long t2 = __shfl_xor_sync(0xffffffffu, chs, o);
            chs = t2 > chs ? t2 : chs;
        }
        if ((tid & 31) == 0) s_max[tid >> 5] = chs;
        __syncthreads();
        if (tid == 0) {
            unsigned long long m = 0ull;
            for (int w = 0; w < (int)blockDim.x / 32; ++w) m = s_max[w] > m ? s_max[w] : m;
            atomicMax(&a.sync->last, m);
        }
        if (!grid_sync(&a.sync->bar, at, nblocks, &s_flag)) failed = true;
        else if (tid == 0) last = __longlong_as_double((long long)ld_relaxed(&a.sync->last));
    }
    if (blockIdx.x == 0 && tid == 0) {
        Ctl* const ctl = a.ctl;
        ctl->ik = done;
        ctl->inner = done_c;
        ctl->cycles = a.itmax > 0 ? cycles : 0;
        ctl->restarts = a.itmax > 0 ? cycles - 1 : 0;
        ctl->bodies = done;
        ctl->last_change = last;
        ctl->converged = conv ? 1 : 0;
        ctl->nonfinite = nonfinite ? 1 : 0;
        ctl->timeout = failed ? 1 : 0;
    }
}

// Start of a solve of the marching kernel: its barrier and slot cleared.
__global__ void k_march_begin(ResSync* rs) {
    rs->bar.word[0] = rs->bar.word[1] = 0ULL;
    rs->bar.err = 0;
    rs->last = 0ULL;
}

}  // namespace ntcfd
