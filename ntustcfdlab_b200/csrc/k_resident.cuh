// k_resident.cuh -- a whole pressure solve (every defect-correction cycle)
// in one persistent cooperative kernel, with the correction e resident in
// shared memory.
//
// The interior rows (j,k) are split into nbj x nbk bricks of balanced sizes;
// CTA b owns brick (b % nbj, b / nbj) and keeps e of both colours for
// its rows in shared memory (colour-split rows of mx entries, see
// ntcfd_common.cuh) with a one-row ring, and the defect d and 1/diag rd of its
// rows when they fit.  The ring rows of a domain boundary stay 0; the others
// hold the neighbour bricks' boundary rows.  A half-sweep runs
//     interior rows -> ring -> edge rows (published) -> CTA barrier.
//
// The ring (k_exchange.cuh).  The owner of an edge cell stores each new value as
// one word with a sequence number into the inbox of the CTA that needs it, and that
// CTA polls the words into its ring: the hand-over costs one trip through L2, which
// the interior rows cover.  An inbox holds one word per ring cell and colour.  A
// CTA publishes a colour only after a CTA barrier that follows its reading of the
// other colour, which its neighbour published after reading the first: no word is
// overwritten unread.  A grid barrier per half-sweep and a copy of the published
// rows afterwards, which this replaces, took 3.4 us of an 8.0 us FP32 sweep at 128^3.
// A sweep takes 6.4 us at 128^3 FP32 (8.0 before), 11.3 FP64 (11.8) and 3.4 us at 40^3
// (5.3): on small grids the hand-over, some 1.5 us per
// half-sweep from a store to its sight by the neighbour, is all that is left; at 128^3
// 56% of the issue slots (FP32; FP64, whose d and rd come from L2, 40%) and 44% of the
// shared-memory pipe are used, and 16 warps wait in turn for shared loads, L2 and the hand-over.
//
// The stop rule (GS.f90:11,53).  A sweep ends the solve when no cell of either colour
// changed by more than zeta.  Every CTA adds the verdict of its red half to a
// counter when that half ends and reads the sum when its black half has ended: one
// red change above zeta anywhere already decides that the solve goes on, so the
// black half's verdicts are waited for only in a sweep whose red half had none.
// The sweep count, the count of correction cycles and the final p += e run inside
// the kernel, and so do the restarts of the defect correction: when a
// cycle ends on its length (cycle_len sweeps), the kernel refreshes the black
// ring, adds e to p and updates d to the FP64 defect of p + e
// (defect_update: d + rdiag sum c e_nb - e, in FP64, from the exact FP32
// values of e), then sweeps on from e = 0.  The first
// defect of the solve comes from k_defect.
//
// A lane updates two cells at a time with every load issued before any
// store: cells t and t + 32 of one row (rows of at most 64 cells per colour,
// or in 64-cell chunks for wider rows; one cell where a last chunk has 32 or fewer: 160x120x120
// FP64 17.5 us a sweep against 19.9 with two throughout), or, in the NARROW instance (rows of
// at most 32 cells per colour), t of two rows.  The row's parity r is a
// template argument of the update, so the east/west neighbours and the second
// cell are immediate offsets of one address.  Loads always read inside the
// shared-memory allocation (or the padded global arrays); a lane past the
// row's last cell stores nothing and leaves the change maximum alone.
//
// Every wait is bounded: a CTA that gives up sets sync->bar.err, the others leave
// the sweep loop at their next wait, and the host reports NTCFD_ETIMEOUT.
#pragma once

#include <type_traits>

#include "k_exchange.cuh"
#include "k_pressure.cuh"
#include "ntcfd_common.cuh"

namespace ntcfd {

// Row shapes of k_sor_resident (Brick::mode): several rows side by side on a warp's lanes; rows of 33
// to 64 cells per colour; a warp per longer row; a warp per 64-cell chunk of a longer row, for bricks of
// few rows (1000x20x16, three or four rows of eight chunks a CTA: FP32 6.7 us a sweep against 7.6 by
// rows), which may be one row thick.
enum { kResNarrow = 0, kResWide1 = 1, kResWide = 2, kResLong = 3 };

struct Brick {
    int nbj, nbk;    // bricks along j and k
    int JB, KB;      // rows of the largest brick
    int mx;          // colour-split row length (compact index m = 0..mx-1)
    int cache_d;     // 1: d of the brick lives in shared memory too
    int cache_rd;    // 1: rd of the brick lives in shared memory too
    int mode;        // kResNarrow, kResWide1 or kResWide (res_mode(nx)); kResLong: wide rows by chunks
    int inbox;       // ring words per CTA and colour
    int deep;        // 1: k_sor_deep (k_resident_deep.cuh)
};

// Cells of a colour in a row: (nx + r) / 2 for parity r; at most (nx + 1) / 2.
__host__ __device__ inline int res_mode(int nx) {
    const int most = (nx + 1) / 2;
    return most <= 32 ? kResNarrow : most <= 64 ? kResWide1 : kResWide;
}

// Rows of a brick with a neighbour, at most.
__host__ __device__ inline int res_edge_rows(int JB, int KB) {
    return JB > 2 && KB > 2 ? 2 * (JB + KB) - 4 : JB * KB;
}
// Bytes of the edge rows' places in the neighbours' inboxes.
inline size_t resident_places(const Brick& b) {
    return (size_t)res_edge_rows(b.JB, b.KB) * (b.mode == kResLong ? 16 : 8);
}

// Dynamic shared memory of k_sor_resident for a brick plan.
template <class Tc>
inline size_t resident_smem(const Brick& b, int nx) {
    const size_t tile = (size_t)(b.JB + 2) * (b.KB + 2) * b.mx;
    const size_t brick = (size_t)b.JB * b.KB * b.mx;
    const size_t arrays = sizeof(Tc) * (2 * tile + 2 * (size_t)(nx + 4) + 2 * (size_t)(b.JB + b.KB) +
                                        (b.cache_d ? 2 * brick : 0) + (b.cache_rd ? 2 * brick : 0));
    // + row table (int4 offsets and four coefficients per row), + the ring list (int2 per
    // ring row), + the edge rows' places, + slack: the loads of a lane past a row's last cell may
    // reach up to 64 elements beyond the tiles
    const size_t rows = (size_t)b.JB * b.KB;
    return ((arrays + 15) & ~size_t(15)) + rows * (16 + 4 * sizeof(Tc)) + 2 * (size_t)(b.JB + b.KB) * 8 +
           resident_places(b) + 64 * sizeof(Tc);
}

// ring words a thread holds in flight (FP64: of three many a brick's ring takes a second round of
// polls, 101x89x105 7.7 us a sweep against 6.8; more than these in FP32 lengthen every round, 256x24x24 3.3
// us a sweep, 4.2 with twelve)
template <class Tc>
constexpr int kFillOf = sizeof(Tc) == 4 ? 6 : 4;

constexpr unsigned int kNanFlag = 1u << 20;   // high-half flag of a CTA whose max |change| was not finite

// Row e of a brick's edge ring (jl or kl on the brick boundary), for e < ne,
// or of its interior, for e >= ne; nj x nk rows, ni = interior rows.
__device__ __forceinline__ void brick_row(int e, int nj, int nk, int ni, int ne, int& jl, int& kl) {
    if (ni == 0) {                       // every row is an edge row
        jl = e % nj + 1;
        kl = e / nj + 1;
    } else if (e >= ne) {                // interior: (nj-2) x (nk-2) rows
        const int q = e - ne;
        jl = q % (nj - 2) + 2;
        kl = q / (nj - 2) + 2;
    } else if (e < 2 * nj) {             // first and last k-row of the brick
        jl = e % nj + 1;
        kl = e < nj ? 1 : nk;
    } else {                             // first and last j-row, inner k
        const int q = e - 2 * nj;
        kl = q % (nk - 2) + 2;
        jl = q < nk - 2 ? 1 : nj;
    }
}

// Everything one half-sweep needs to know about a row.
template <class Tc>
struct ResRow {
    const Tc* O;      // other colour, tile row start (shared)
    Tc* W;            // own colour, tile row start (shared)
    const Tc* D;      // d of the row: brick row start (shared) or global row start
    const Tc* R;      // rd of the row, likewise
    Tc cN, cS, cF, cB;
    int par;          // (j + k) & 1 of the row
    unsigned long long *pubA, *pubB;   // an edge row's words in its neighbours' inboxes (t = 0; null: none)
    unsigned long long *pubC, *pubD;   // (FOUR)
};

// The loaded operands of one cell.
template <class Tc>
struct ResIn {
    Tc oE, oW, oN, oS, oF, oB, e0, d, rd;
};

// Loads of cell t of a row, at own index m = t + 2 - parity, all from shared memory:
// the tile's ring holds the neighbour bricks' rows of the other colour (fill).
// The east and west neighbours sit at t + 2 and t + 1 whatever the parity.
// d may be rewritten inside the launch by this CTA
// only: a plain (L1-coherent) load when it is global.
template <class Tc, bool CD, bool CR>
__device__ __forceinline__ ResIn<Tc> res_load(const ResRow<Tc>& w, int t, int m, int mx, int plane) {
    ResIn<Tc> x;
    const Tc* o = w.O + m;
    x.oE = w.O[t + 2];
    x.oW = w.O[t + 1];
    x.oN = o[mx];
    x.oS = o[-mx];
    x.oF = o[plane];
    x.oB = o[-plane];
    x.e0 = w.W[m];
    x.d = CD ? w.D[m] : __ldca(w.D + m);
    if (CR) x.rd = w.R[m];
    else if (!CD) x.rd = __ldg(w.R + m);
    return x;
}

// The update of a loaded cell t of a row; stores e and takes the change into the
// maximum only when ok.  A cell of an EDGE row goes to the neighbours' inboxes too
// (ring: a cell of the ring; 0 where a row is a cell shorter than the ring).
//
// Where d has room on the chip and rd has none, rd is formed from the coefficients: 7.7 us a
// sweep against 8.4 with rd from L2 on 100x150x150 FP32, 8.2 against 9.8 on 112^3
// FP64.  Where d comes from L2 as well, rd does too (formed: 64x128x256 FP64 13.0 us
// against 12.4).
template <class Tc, bool EDGE, bool FORM, bool FOUR, class B>
__device__ __forceinline__ void res_finish(const ResIn<Tc>& x, const ResRow<Tc>& w, int t, int m, Tc cE, Tc cW, Tc om,
                                           bool ok, bool ring, unsigned int seq, B& ch) {
    Tc e1;
    const Tc rd = FORM ? rdiag_near(((cE + cW) + (w.cN + w.cS)) + (w.cF + w.cB)) : x.rd;
    const Tc diff = sor_update(cE, x.oE, cW, x.oW, w.cN, x.oN, w.cS, x.oS, w.cF, x.oF, w.cB, x.oB, rd, x.d,
                               x.e0, om, &e1);
    if (ok) {
        w.W[m] = e1;
        const B db = abs_bits(diff);
        ch = db > ch ? db : ch;
    }
    if (EDGE) {
        using Word = RingWord<Tc>;
        const Tc v = ok ? e1 : Tc(0);
        if (ring && w.pubA) Word::store(w.pubA + t * Word::n, v, seq);
        if (ring && w.pubB) Word::store(w.pubB + t * Word::n, v, seq);
        if (FOUR && ring && w.pubC) Word::store(w.pubC + t * Word::n, v, seq);
        if (FOUR && ring && w.pubD) Word::store(w.pubD + t * Word::n, v, seq);
    }
}

template <class Tc, int NT, bool CD, bool CR, int MODE>
__global__ void __launch_bounds__(NT, 1)
k_sor_resident(Geom g, SorCoef<Tc> sc, Brick br, double* __restrict__ p,
               Tc* __restrict__ dRg, Tc* __restrict__ dBg, const Tc* __restrict__ rdRg,
               const Tc* __restrict__ rdBg, Ctl* ctl, ResSync* sync, unsigned long long* boxes,
               double omega, double zeta, int itmax, int cycle_len, int check_every) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using B = decltype(abs_bits(Tc(0)));
    constexpr int kFill = kFillOf<Tc>;
    using Word = RingWord<Tc>;
    __shared__ int s_flag, s_fail[2], s_nan[2];   // by the sweep's parity, so that a thread ahead writes the other
    // verdicts of the sweep (CTAs above zeta, kNanFlag per NaN): red half, black half (of the
    // sweep before until this one's is waited for)
    __shared__ uint2 s_vd;
    __shared__ unsigned int s_prev[2][4];         // high halves of the counters at their last use
    __shared__ B s_red_max[NT / 32];
    const int JB = br.JB, KB = br.KB, mx = br.mx;
    const int RS = JB + 2;                    // rows per k-plane of the tile
    const int plane = RS * mx;
    const int tile = plane * (KB + 2);
    const int brick = JB * KB * mx;
    // shared memory: e red, e black (tile with halo), coefficients cE, cW (index
    // i+1, i = -1..nx+2), cN, cS of the brick's rows, cF, cB of its planes, then d
    // red/black and rd red/black of the brick when cached, then the row table
    Tc* const S0 = reinterpret_cast<Tc*>(smem_raw);
    Tc* const S1 = S0 + tile;
    Tc* const cEs = S1 + tile + 1;
    Tc* const cWs = cEs + (g.nx + 4);
    Tc* const cNs = cEs + 2 * (g.nx + 4) - 1;
    Tc* const cSs = cNs + JB;
    Tc* const cFs = cSs + JB;
    Tc* const cBs = cFs + KB;
    Tc* const D0 = cBs + KB;
    Tc* const D1 = D0 + brick;
    Tc* const R0 = CD ? D1 + brick : D0;
    Tc* const R1 = R0 + brick;
    Tc* const arrays_end = CR ? R1 + brick : (CD ? D1 + brick : D0);
    // row table: per row of the brick, in sweep order (edge rows first), the tile row
    // start, the brick row start of d/rd, the global colour-split row start and
    // (j+k)&1; the row's cN, cS, cF, cB; of the edge rows their places in the neighbours'
    // inboxes.  Then the ring: per row of a neighbour brick (inbox order) its tile row start and (j+k)&1.
    const size_t toff = ((size_t)((unsigned char*)arrays_end - smem_raw) + 15) & ~size_t(15);
    int4* const rowT = reinterpret_cast<int4*>(smem_raw + toff);
    Tc* const rowC = reinterpret_cast<Tc*>(rowT + JB * KB);
    using Places = std::conditional_t<MODE == kResLong, int4, int2>;
    Places* const pubT = reinterpret_cast<Places*>(rowC + 4 * JB * KB);
    int2* const ringT = reinterpret_cast<int2*>(pubT + res_edge_rows(JB, KB));
    constexpr int NWARP = NT / 32;
    // an update of its own for each parity of a row (the warp's rows have one each): without the selects by
    // parity narrow rows take 11.3 us a sweep against 12.6 (48x192x187 FP32), 12.0 against 13.2
    // (33x134x264 FP64), 128^3 FP64 11.2 against 11.4; other wide rows are slower so (112^3 FP64 8.7
    // against 8.4, FP32 6.9 against 6.7)
    constexpr bool kParity = MODE == kResNarrow || (MODE == kResWide1 && sizeof(Tc) == 8 && !CD);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tid = threadIdx.x;

    const int bj = blockIdx.x % br.nbj, bk = blockIdx.x / br.nbj;
    const int j0 = 1 + brick_start(bj, g.ny, br.nbj), nj = 1 + brick_start(bj + 1, g.ny, br.nbj) - j0;
    const int k0 = 1 + brick_start(bk, g.nz, br.nbk), nk = 1 + brick_start(bk + 1, g.nz, br.nbk) - k0;
    const bool jlo = bj > 0, jhi = bj < br.nbj - 1, klo = bk > 0, khi = bk < br.nbk - 1;   // neighbouring bricks
    const bool multi = gridDim.x > 1;
    const int ys = g.mxp, zs = (int)g.mz;   // colour-split row and plane pitch
    // cells of a colour in a row of parity r
    const int nown0 = g.nx / 2, nown1 = (g.nx + 1) / 2;

    for (int q = tid; q < 2 * tile; q += NT) S0[q] = Tc(0);
    for (int i = tid - 1; i <= g.nx + 2; i += NT) {
        cEs[i] = sc.cE[i];
        cWs[i] = sc.cW[i];
    }
    for (int q = tid; q < JB; q += NT) {
        const int j = min(j0 + q, g.ny);
        cNs[q] = sc.cN[j];
        cSs[q] = sc.cS[j];
    }
    for (int q = tid; q < KB; q += NT) {
        const int k = min(k0 + q, g.nz);
        cFs[q] = sc.cF[k];
        cBs[q] = sc.cB[k];
    }
    const int nrows = nj * nk;
    const int ni = (nj > 2 && nk > 2) ? (nj - 2) * (nk - 2) : 0;   // interior rows
    const int ne = nrows - ni;                                       // edge rows
    // the ring rows in the order of the inbox: faces j-low, j-high (nk rows each), k-low,
    // k-high (nj rows each), those without a neighbour left out
    const int fj = (jlo ? nk : 0) + (jhi ? nk : 0), nring = fj + (klo ? nj : 0) + (khi ? nj : 0);
    for (int q = tid; q < nring; q += NT) {
        int jl, kl;
        if (q < fj) {
            kl = q % nk + 1;
            jl = jlo && q < nk ? 0 : nj + 1;
        } else {
            const int r = q - fj;
            jl = r % nj + 1;
            kl = klo && r < nj ? 0 : nk + 1;
        }
        ringT[q] = make_int2((kl * RS + jl) * mx, (j0 + jl - 1 + k0 + kl - 1) & 1);
    }
    // planes of the neighbours along k (those along j have this brick's)
    const int nkl = klo ? k0 - 1 - brick_start(bk - 1, g.nz, br.nbk) : 0;
    const int nkh = khi ? brick_start(bk + 2, g.nz, br.nbk) - brick_start(bk + 1, g.nz, br.nbk) : 0;
    for (int er = tid; er < nrows; er += NT) {
        int jl, kl;
        brick_row(er, nj, nk, ni, ne, jl, kl);
        const int j = j0 + jl - 1, k = k0 + kl - 1;
        rowT[er] = make_int4((kl * RS + jl) * mx, ((kl - 1) * JB + (jl - 1)) * mx, ys * (j + 1) + zs * (k + 1),
                             (j + k) & 1);
        rowC[4 * er + 0] = sc.cN[j];
        rowC[4 * er + 1] = sc.cS[j];
        rowC[4 * er + 2] = sc.cF[k];
        rowC[4 * er + 3] = sc.cB[k];
        if (er >= ne) continue;
        // the row's ring row in a neighbour: at most one along j and one along k (a brick
        // that has neighbours on both sides of a direction is two rows thick or more)
        auto place = [&](int cta, int ring_row) { return cta * 2 * br.inbox + ring_row * nown1; };
        const int me = (int)blockIdx.x;
        const bool toJl = jl == 1 && jlo, toJh = jl == nj && jhi, toKl = kl == 1 && klo, toKh = kl == nk && khi;
        const int pJl = place(me - 1, (bj > 1 ? nk : 0) + kl - 1);       // the j-high face of brick bj - 1
        const int pJh = place(me + 1, kl - 1);                           // the j-low face of brick bj + 1
        const int pKl = place(me - br.nbj, (jlo ? nkl : 0) + (jhi ? nkl : 0) + (bk > 1 ? nj : 0) + jl - 1);
        const int pKh = place(me + br.nbj, (jlo ? nkh : 0) + (jhi ? nkh : 0) + jl - 1);
        const int pj = toJl ? pJl : toJh ? pJh : -1, pk = toKl ? pKl : toKh ? pKh : -1;
        if constexpr (MODE == kResLong) pubT[er] = make_int4(toJl ? pJl : -1, toJh ? pJh : -1, toKl ? pKl : -1, toKh ? pKh : -1);
        else pubT[er] = pj >= 0 ? make_int2(pj, pk) : make_int2(pk, -1);
    }
    if (tid == 0) {
        s_fail[0] = s_fail[1] = s_nan[0] = s_nan[1] = 0;
        s_vd = make_uint2(0u, 0u);
    }
    if (tid < 8) s_prev[tid >> 2][tid & 3] = 0u;
    if (CD || CR) {
        // d (the solve's first defect, from k_defect) and rd of the brick: one warp per
        // row, lanes along m
        for (int row = warp; row < nrows; row += NWARP) {
            const int jl = row % nj, kl = row / nj;
            const long long gq0 = spl(g, 0, j0 + jl, k0 + kl);
            const int sq0 = (kl * JB + jl) * mx;
            for (int m = lane; m < mx; m += 32) {
                if (CD) {
                    D0[sq0 + m] = dRg[gq0 + m];
                    D1[sq0 + m] = dBg[gq0 + m];
                }
                if (CR) {
                    R0[sq0 + m] = rdRg[gq0 + m];
                    R1[sq0 + m] = rdBg[gq0 + m];
                }
            }
        }
    }
    __syncthreads();
    // the lane's cell t in the narrow form, and its row among the rpw side by side
    const int rpw = MODE == kResNarrow ? 32 / nown1 : 1;
    // (in FP64 the lanes left over go on past the end of the last row: from a row's start they would
    // meet the other lanes' banks)
    const int most = sizeof(Tc) == 8 ? rpw - 1 : rpw;
    const int sub = MODE == kResNarrow ? min(lane / nown1, most) : 0, lt = lane - sub * nown1;
    const bool lane_in = sub < rpw && lt < nown1;
    // lane coefficients of the one- and two-row instances: the cells t = lt (and
    // t = lt + 32) of a row of parity r sit at i = 2t + 2 - r (past the row's end
    // they read other table entries, never used)
    Tc cEr[2][2], cWr[2][2];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = 2 * (lt + 32 * h) + 2 - r;
            cEr[r][h] = MODE >= kResWide ? Tc(0) : cEs[min(i, g.nx + 2)];
            cWr[r][h] = MODE >= kResWide ? Tc(0) : cWs[min(i, g.nx + 2)];
        }

    const unsigned int nblocks = gridDim.x;
    const unsigned int seq0 = sync->seq;
    const bool ctrl = multi && tid == NT / 2;   // the thread that talks to the counters
    const int ik0 = ctl->ik;
    const Tc om = (Tc)omega;
    int done = 0;        // sweeps of this launch
    int done_c = 0;      // sweeps of the current cycle
    int restarts = 0;
    bool conv = false, nonfinite = false, failed = false;
    bool tested = false, prev_tested = false;   // a stop test ran; in the sweep before
    B chs = B(0);        // this thread's max |change| of the last sweep
    double last = 0.0;

    // p += e over the brick (natural <- shared memory); one warp per pair of rows,
    // lanes along i, 8 values of p in flight per lane
    auto add_e_to_p = [&]() {
        constexpr int U = 4;
        for (int row = 2 * warp; row < nrows; row += 2 * NWARP) {
            for (int i0 = 1; i0 <= g.nx; i0 += 32 * U) {
                double pv[2][U];
                long long c0[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int rr = min(row + h, nrows - 1);
                    c0[h] = nat(g, 0, j0 + rr % nj, k0 + rr / nj);
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int i = i0 + lane + 32 * u;
                        if (i <= g.nx) pv[h][u] = p[c0[h] + i];
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (row + h >= nrows) continue;
                    const int jl = (row + h) % nj + 1, kl = (row + h) / nj + 1;
                    const int j = j0 + jl - 1, k = k0 + kl - 1;
                    const int sr = (kl * RS + jl) * mx;
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int i = i0 + lane + 32 * u;
                        if (i <= g.nx)
                            p[c0[h] + i] = pv[h][u] + (double)(((i + j + k) & 1) ? S1 : S0)[sr + ((i + 2) >> 1)];
                    }
                }
            }
        }
    };

    struct DefIn {
        Tc* D;          // d of the row: shared (CD) or global
        double* pr;     // natural row of p, i = 0
        int nown, mA, iA;
        Tc oEA, oWA, oNA, oSA, oFA, oBA, oEB, oWB, oNB, oSB, oFB, oBB, eA, eB, dA, dB;
        double cEA, cWA, cEB, cWB, cN, cS, cF, cB, pA, pB;
    };
    // every load of the cells t0 + lane and t0 + lane + 32 of task rc = 2 * row + colour
    auto def_load = [&](int rc, int t0) {
        DefIn x;
        const int row = rc >> 1, c = rc & 1;
        const int jl = row % nj + 1, kl = row / nj + 1;
        const int j = j0 + jl - 1, k = k0 + kl - 1;
        const int r = ((j + k) ^ c) & 1;
        x.nown = r ? nown1 : nown0;
        x.cN = g.cN[j]; x.cS = g.cS[j]; x.cF = g.cF[k]; x.cB = g.cB[k];
        const int sr = (kl * RS + jl) * mx, dr = ((kl - 1) * JB + (jl - 1)) * mx;
        const Tc* O = (c ? S0 : S1) + sr;         // the other colour's tile row
        const Tc* Wt = (c ? S1 : S0) + sr;        // this colour's
        x.D = CD ? (c ? D1 : D0) + dr : (c ? dBg : dRg) + spl(g, 0, j, k);
        x.pr = p + nat(g, 0, j, k);
        const int tA = t0 + lane;
        const int mA = tA + 2 - r, mB = mA + 32;
        x.mA = mA;
        x.iA = 2 * tA + 2 - r;
        const int iAc = min(x.iA, g.nx + 2), iBc = min(x.iA + 64, g.nx + 2);
        x.oEA = O[mA + r]; x.oWA = O[mA - 1 + r]; x.oNA = O[mx + mA]; x.oSA = O[mA - mx];
        x.oFA = O[plane + mA]; x.oBA = O[mA - plane];
        x.oEB = O[mB + r]; x.oWB = O[mB - 1 + r]; x.oNB = O[mx + mB]; x.oSB = O[mB - mx];
        x.oFB = O[plane + mB]; x.oBB = O[mB - plane];
        x.eA = Wt[mA]; x.eB = Wt[mB];
        x.dA = x.D[mA]; x.dB = x.D[mB];
        x.cEA = g.cE[iAc]; x.cWA = g.cW[iAc]; x.cEB = g.cE[iBc]; x.cWB = g.cW[iBc];
        x.pA = x.pr[x.iA]; x.pB = x.pr[x.iA + 64];
        return x;
    };
    auto def_finish = [&](const DefIn& x, int t0) {
        const double dnA = defect_update(x.cEA, x.oEA, x.cWA, x.oWA, x.cN, x.oNA, x.cS, x.oSA, x.cF, x.oFA, x.cB,
                                         x.oBA, x.dA, x.eA);
        const double dnB = defect_update(x.cEB, x.oEB, x.cWB, x.oWB, x.cN, x.oNB, x.cS, x.oSB, x.cF, x.oFB, x.cB,
                                         x.oBB, x.dB, x.eB);
        const int tA = t0 + lane;
        if (tA < x.nown) {
            x.D[x.mA] = (Tc)dnA;
            x.pr[x.iA] = x.pA + (double)x.eA;
        }
        if (tA + 32 < x.nown) {
            x.D[x.mA + 32] = (Tc)dnB;
            x.pr[x.iA + 64] = x.pB + (double)x.eB;
        }
    };
    // Restart of a correction cycle: d of every cell of the brick becomes the FP64
    // defect of p + e (defect_update), from the tiles (both rings current), and the
    // cycle's e goes to p in the same pass (add_e_to_p takes only the last cycle's);
    // a warp per row and colour ("task"), lane t takes the cells t and t + 32 of
    // each 64-cell chunk (consecutive m: each shared-memory load of the warp reads
    // one tile without bank conflicts).  FP32 rows of 33-64 cells per colour (the
    // kResWide1 instance) go two tasks at a time, every load of both (p from L2
    // among them) issued before the FP64 arithmetic of either.  A lane past the row's last cell reads inside the
    // shared allocation, the padded d arrays and the natural p array (ghost rows
    // and planes follow the brick's) and stores nothing.
    auto update_defect = [&]() {
        // (FP64, whose restarts are rare, and the other row shapes keep one task at a
        // time: the pair makes those instances spill)
        if (sizeof(Tc) == 4 && MODE == kResWide1) {
            for (int rc = warp; rc < 2 * nrows; rc += 2 * NWARP) {
                const bool two = rc + NWARP < 2 * nrows;
                const DefIn xa = def_load(rc, 0);
                const DefIn xb = def_load(two ? rc + NWARP : rc, 0);
                def_finish(xa, 0);
                if (two) def_finish(xb, 0);
            }
        } else {
            for (int rc = warp; rc < 2 * nrows; rc += NWARP) {
                const int row = rc >> 1;
                const int r = ((j0 + row % nj + k0 + row / nj) ^ (rc & 1)) & 1;
                const int nown = r ? nown1 : nown0;
                for (int t0 = 0; t0 < nown; t0 += 64) {
                    const DefIn xa = def_load(rc, t0);
                    def_finish(xa, t0);
                }
            }
        }
    };
    auto zero_tile = [&]() {
        for (int q = tid; q < 2 * tile; q += NT) S0[q] = Tc(0);
    };


    // ---- the ring of colour oc from this CTA's inbox, words numbered seq: kFill words per
    // thread in flight, polled until they carry the number.  A CTA barrier follows.
    const unsigned int mH = 0xffffffffu / (unsigned)nown1 + 1u;   // q / nown1, exact for q * nown1 < 2^32
    const int ring_tot = nring * nown1;
    const size_t boxw = (size_t)br.inbox * Word::n;               // 8-byte words of a colour
    auto fill = [&](int oc, unsigned int seq, int par) {
        Tc* const O = oc ? S1 : S0;
        const unsigned long long* const bx = boxes + ((size_t)blockIdx.x * 2 + oc) * boxw;
        for (int q0 = 0; q0 < ring_tot; q0 += NT * kFill) {
            Word w[kFill];
#pragma unroll
            for (int u = 0; u < kFill; ++u)
                w[u].load(bx + (size_t)min(q0 + tid + NT * u, ring_tot - 1) * Word::n);
            for (unsigned int polls = 0;; ++polls) {
                bool all = true;
#pragma unroll
                for (int u = 0; u < kFill; ++u) all = all && w[u].has(seq);
                if (all) break;
                if ((polls & 255u) == 255u && ring_lost(sync, polls)) {
                    s_fail[par] = 1;
                    break;
                }
#pragma unroll
                for (int u = 0; u < kFill; ++u)
                    w[u].load(bx + (size_t)min(q0 + tid + NT * u, ring_tot - 1) * Word::n);
            }
#pragma unroll
            for (int u = 0; u < kFill; ++u) {
                const int q = q0 + tid + NT * u;
                if (q >= ring_tot) continue;
                const unsigned int r = __umulhi((unsigned)q, mH);
                const int2 rr = ringT[r];
                // cell t of the row sits at m = t + 2 - parity
                O[rr.x + (q - (int)r * nown1) + 2 - (rr.y ^ oc)] = w[u].value();
            }
        }
    };

    // ---- one half-sweep of colour c over rows [e0r, e1r) (edge rows: EDGE)
    const int nch = (nown1 + 63) / 64;                            // chunks of a row (kResLong)
    const int row0 = warp / nch, chunk0 = warp - row0 * nch, rowstep = NWARP / nch, chunkstep = NWARP - rowstep * nch;
    auto rows_pass = [&](auto edge_tag, int c, int e0r, int e1r, unsigned int seq, B& ch) {
        constexpr bool EDGE = decltype(edge_tag)::value;
        Tc* const W = c ? S1 : S0;
        const Tc* const O = c ? S0 : S1;
        unsigned long long* const Ec = boxes + (size_t)c * boxw;
        const Tc* const Dg = c ? dBg : dRg;
        const Tc* const Rg = c ? rdBg : rdRg;
        const Tc* const Ds = c ? D1 : D0;
        const Tc* const Rs = c ? R1 : R0;
        auto row_of = [&](int er) {
            const int4 rt = rowT[er];
            ResRow<Tc> w;
            w.O = O + rt.x;
            w.W = W + rt.x;
            w.D = CD ? Ds + rt.y : Dg + rt.z;
            w.R = CR ? Rs + rt.y : Rg + rt.z;
            if constexpr (sizeof(Tc) == 4) {
                const float4 c4 = *reinterpret_cast<const float4*>(rowC + 4 * er);
                w.cN = c4.x; w.cS = c4.y; w.cF = c4.z; w.cB = c4.w;
            } else {
                const double2 a2 = *reinterpret_cast<const double2*>(rowC + 4 * er);
                const double2 b2 = *reinterpret_cast<const double2*>(rowC + 4 * er + 2);
                w.cN = a2.x; w.cS = a2.y; w.cF = b2.x; w.cB = b2.y;
            }
            w.par = rt.w;
            if (EDGE) {
                const Places pb = pubT[er];
                w.pubA = pb.x >= 0 ? Ec + (size_t)pb.x * Word::n : nullptr;
                w.pubB = pb.y >= 0 ? Ec + (size_t)pb.y * Word::n : nullptr;
                if constexpr (MODE == kResLong) {
                    w.pubC = pb.z >= 0 ? Ec + (size_t)pb.z * Word::n : nullptr;
                    w.pubD = pb.w >= 0 ? Ec + (size_t)pb.w * Word::n : nullptr;
                }
            }
            return w;
        };
        if constexpr (MODE == kResNarrow) {
            // rows of at most 32 cells per colour: a warp takes 2 rpw rows at a time, rpw side by
            // side over the lanes (rpw = 32 / nown1), twice
            auto pair = [&](const ResRow<Tc>& wA, const ResRow<Tc>& wB, int rA, int rB, bool inA, bool inB) __attribute__((always_inline)) {
                const int mA = lt + 2 - rA, mB = lt + 2 - rB;
                const ResIn<Tc> xA = res_load<Tc, CD, CR>(wA, lt, mA, mx, plane);
                const ResIn<Tc> xB = res_load<Tc, CD, CR>(wB, lt, mB, mx, plane);
                res_finish<Tc, EDGE, CD && !CR, false>(xA, wA, lt, mA, rA ? cEr[1][0] : cEr[0][0], rA ? cWr[1][0] : cWr[0][0], om,
                                     inA && lt < (rA ? nown1 : nown0), inA, seq, ch);
                res_finish<Tc, EDGE, CD && !CR, false>(xB, wB, lt, mB, rB ? cEr[1][0] : cEr[0][0], rB ? cWr[1][0] : cWr[0][0], om,
                                     inB && lt < (rB ? nown1 : nown0), inB, seq, ch);
            };
            if (rpw == 1) {
                for (int er = e0r + 2 * warp; er < e1r; er += 2 * NWARP) {
                    const bool inB = lane_in && er + 1 < e1r;
                    const ResRow<Tc> wA = row_of(er), wB = row_of(er + 1 < e1r ? er + 1 : er);
                    const int rA = (wA.par ^ c) & 1, rB = (wB.par ^ c) & 1;
                    if (rA == 0) {
                        if (rB == 0) pair(wA, wB, 0, 0, lane_in, inB);
                        else pair(wA, wB, 0, 1, lane_in, inB);
                    } else {
                        if (rB == 0) pair(wA, wB, 1, 0, lane_in, inB);
                        else pair(wA, wB, 1, 1, lane_in, inB);
                    }
                }
            } else {
                for (int er = e0r + 2 * rpw * warp + sub; er < e1r + sub; er += 2 * rpw * NWARP) {
                    const int eB = er + rpw;
                    const bool inA = lane_in && er < e1r, inB = lane_in && eB < e1r;
                    const ResRow<Tc> wA = row_of(er < e1r ? er : e0r), wB = row_of(eB < e1r ? eB : e0r);
                    pair(wA, wB, (wA.par ^ c) & 1, (wB.par ^ c) & 1, inA, inB);
                }
            }
        } else if constexpr (MODE == kResWide1) {
            for (int er = e0r + warp; er < e1r; er += NWARP) {
                const ResRow<Tc> w = row_of(er);
                // cells t = lane (always in the row: it holds more than 32) and lane + 32
                auto one = [&](int r) __attribute__((always_inline)) {
                    const int nown = r ? nown1 : nown0, m = lane + 2 - r;
                    const ResIn<Tc> xA = res_load<Tc, CD, CR>(w, lane, m, mx, plane);
                    const ResIn<Tc> xB = res_load<Tc, CD, CR>(w, lane + 32, m + 32, mx, plane);
                    res_finish<Tc, EDGE, CD && !CR, false>(xA, w, lane, m, r ? cEr[1][0] : cEr[0][0], r ? cWr[1][0] : cWr[0][0], om, true,
                                         true, seq, ch);
                    res_finish<Tc, EDGE, CD && !CR, false>(xB, w, lane + 32, m + 32, r ? cEr[1][1] : cEr[0][1], r ? cWr[1][1] : cWr[0][1],
                                         om, lane + 32 < nown, lane + 32 < nown1, seq, ch);
                };
                const int r = (w.par ^ c) & 1;
                if (kParity && r) one(1);
                else if (kParity) one(0);
                else one(r);
            }
        } else {
            // the cells t0 + lane, and with `two` t0 + 32 + lane, of a row
            auto chunk = [&](auto two, const ResRow<Tc>& w, int t0) __attribute__((always_inline)) {
                constexpr bool TWO = decltype(two)::value;
                const int r = (w.par ^ c) & 1;
                const int nown = r ? nown1 : nown0;
                const int tA = t0 + lane, m = tA + 2 - r;
                const ResIn<Tc> xA = res_load<Tc, CD, CR>(w, tA, m, mx, plane);
                ResIn<Tc> xB;
                if (TWO) xB = res_load<Tc, CD, CR>(w, tA + 32, m + 32, mx, plane);
                const int iA = min(2 * tA + 2 - r, g.nx + 2), iB = min(iA + 64, g.nx + 2);
                const Tc eA = cEs[iA], wA = cWs[iA], eB = cEs[iB], wB = cWs[iB];
                res_finish<Tc, EDGE, CD && !CR, MODE == kResLong>(xA, w, tA, m, eA, wA, om, tA < nown, tA < nown1, seq, ch);
                if (TWO) res_finish<Tc, EDGE, CD && !CR, MODE == kResLong>(xB, w, tA + 32, m + 32, eB, wB, om, tA + 32 < nown, tA + 32 < nown1, seq, ch);
            };
            if constexpr (MODE == kResLong) {
                // a warp per 64-cell chunk of a row
                int q = chunk0;
                for (int er = e0r + row0; er < e1r; er += rowstep) {
                    chunk(std::true_type{}, row_of(er), 64 * q);
                    if ((q += chunkstep) >= nch) {
                        q -= nch;
                        ++er;
                    }
                }
            } else {
                // a warp per row; of a last chunk of 32 cells or fewer only the first half
                for (int er = e0r + warp; er < e1r; er += NWARP) {
                    const ResRow<Tc> w = row_of(er);
                    int t0 = 0;
                    for (; t0 + 32 < nown1; t0 += 64) chunk(std::true_type{}, w, t0);
                    if (t0 < nown1) chunk(std::false_type{}, w, t0);
                }
            }
        }
    };
    using EdgeT = std::integral_constant<bool, true>;
    using InnerT = std::integral_constant<bool, false>;

    // a change above zeta, NaN included: FP32 changes against the largest float <= zeta
    const float zf = __double2float_rd(zeta);
    auto above = [&](B ch) {
        if constexpr (sizeof(Tc) == 4) return !(__uint_as_float(ch) <= zf);
        else return !(__longlong_as_double((long long)ch) <= zeta);
    };
    auto verdict = [&](int any, int par) {
        return 1ull | (unsigned long long)((any ? 1u : 0u) + (s_nan[par] ? kNanFlag : 0u)) << 32;
    };
    constexpr B kInf = sizeof(Tc) == 4 ? (B)0x7f800000u : (B)kInfBits;

  for (;;) {
    done_c = 0;
#pragma unroll 1
    for (int s = 0; ik0 + done + s < itmax && s < cycle_len; ++s) {
        const int sg = done + s, par = sg & 1;      // sweep of this launch
        const unsigned int target = nblocks * (unsigned)((sg >> 2) + 1);
        const int ik = ik0 + sg + 1;
        const bool test = check_every == 1 || ik >= itmax || ik % check_every == 0;
        B ch = B(0);                                // over both colours
        unsigned int vr = 0u, vb = 0u;              // verdicts: CTAs with a red, a black change above zeta
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
            const unsigned int seq = seq0 + 2u * (unsigned)sg + 1u + (unsigned)c;
            B cc = B(0);
            // the interior rows read only this brick's values; the ring (0 in a cycle's first
            // half-sweep), the edge rows (published)
            rows_pass(InnerT{}, c, ne, nrows, seq, cc);
            if (multi) {
                if (c || s > 0) fill(1 - c, seq - 1u, par);
                __syncthreads();
                if (s_fail[par]) {
                    failed = true;
                    break;
                }
            }
            // the counters' first look, a trip through L2 ahead of its use
            unsigned long long wr = 0ull, wb = 0ull;
            if (c && ctrl) {
                wr = ld_relaxed(&sync->cnt[0][sg & 3]);
                wb = ld_relaxed(&sync->cnt[1][(sg + 3) & 3]);
            }
            rows_pass(EdgeT{}, c, 0, ne, seq, cc);
            if (cc >= kInf) s_nan[par] = 1;
            if (c && ctrl) {
                // the red half's verdicts, and whether the sweep before met a NaN in its black half
                if ((int)((unsigned int)wr - target) < 0 &&
                    !count_wait(&sync->cnt[0][sg & 3], target, &sync->bar.err, &wr))
                    s_fail[par] = 1;
                // every verdict of that half counts: a late one would be taken for the next use of its counter
                const unsigned int before = nblocks * (unsigned)(((sg + 3) >> 2));
                if ((int)((unsigned int)wb - before) < 0 &&
                    !count_wait(&sync->cnt[1][(sg + 3) & 3], before, &sync->bar.err, &wb))
                    s_fail[par] = 1;
                const unsigned int h0 = (unsigned int)(wr >> 32), h1 = (unsigned int)(wb >> 32);
                s_vd = make_uint2(h0 - s_prev[0][sg & 3], sg > 0 ? h1 - s_prev[1][(sg + 3) & 3] : 0u);
                s_prev[0][sg & 3] = h0;
                if (sg > 0) s_prev[1][(sg + 3) & 3] = h1;
            }
            const int any = __syncthreads_or(above(cc));
            if (ctrl) red_add_relaxed(&sync->cnt[c][sg & 3], verdict(any, par));
            (c ? vb : vr) = any ? 1u : 0u;
            ch = cc > ch ? cc : ch;
        }
        if (failed) break;
        if (s_fail[par]) {
            failed = true;
            break;
        }
        if (multi) {
            const uint2 vd = s_vd;
            if (prev_tested && vd.y >= kNanFlag) {
                nonfinite = true;                   // met in the sweep before
                break;
            }
            vr = vd.x;
        } else if (s_nan[par]) {
            vr = kNanFlag;
        }
        chs = ch;
        done_c = s + 1;
        prev_tested = test;
        if (test) {
            tested = true;
            if (multi && vr < kNanFlag && (vr == 0u || ik >= itmax)) {
                __syncthreads();                    // s_vd has been read
                if (ctrl) {
                    unsigned long long w = 0ull;
                    if (!count_wait(&sync->cnt[1][sg & 3], target, &sync->bar.err, &w)) s_fail[par] = 1;
                    s_vd.y = (unsigned int)(w >> 32) - s_prev[1][sg & 3];
                }
                __syncthreads();
                if (s_fail[par]) {
                    failed = true;
                    break;
                }
                vb = s_vd.y;
            }
            nonfinite = vr >= kNanFlag || vb >= kNanFlag;
            conv = vr == 0u && vb == 0u;
            if (conv || nonfinite) break;
        }
    }
    done += done_c;
    // another cycle only when this one ended on its length
    if (failed || conv || nonfinite || done_c < cycle_len || ik0 + done >= itmax) break;
    // restart: the black ring once more (the neighbours' final black rows; the red one is
    // current), d = the FP64 defect of p + e and p += e in one pass, e = 0
    if (multi) {
        fill(1, seq0 + 2u * (unsigned)done, done & 1);
        __syncthreads();
        if (s_fail[done & 1]) {
            failed = true;
            break;
        }
    }
    update_defect();
    __syncthreads();
    zero_tile();
    __syncthreads();
    ++restarts;
  }
    add_e_to_p();
    // the max |change| of the last (tested) sweep
    if (!failed && tested && done > 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const B t2 = __shfl_xor_sync(0xffffffffu, chs, o);
            chs = t2 > chs ? t2 : chs;
        }
        if (lane == 0) s_red_max[warp] = chs;
        __syncthreads();
        if (tid == 0) {
            B b2 = B(0);
            for (int q = 0; q < NWARP; ++q) b2 = s_red_max[q] > b2 ? s_red_max[q] : b2;
            if (multi) atomicMax(&sync->last, widen_bits(b2));
            else last = __longlong_as_double((long long)widen_bits(b2));
        }
        if (multi) {
            GridPlace at;
            if (!grid_sync(&sync->bar, at, nblocks, &s_flag)) failed = true;
            else if (tid == 0) last = __longlong_as_double((long long)ld_relaxed(&sync->last));
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        sync->seq = seq0 + (failed ? 1u << 24 : 2u * (unsigned)done + 4u);
        ctl->ik = ik0 + done;
        ctl->inner = done_c;
        ctl->cycles += restarts + (itmax > 0 ? 1 : 0);   // the launch's cycles, the last included
        ctl->restarts += restarts;
        ctl->bodies += done;
        if (done > 0) ctl->last_change = last;
        if (conv) ctl->converged = 1;
        if (nonfinite) ctl->nonfinite = 1;
        if (failed) ctl->timeout = 1;
    }
}

}  // namespace ntcfd
