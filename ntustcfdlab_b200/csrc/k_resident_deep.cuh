// k_resident_deep.cuh -- the resident pressure solve (k_resident.cuh) for grids of small
// bricks, with one hand-over between CTAs per sweep instead of two.
//
// A hand-over costs some 1.5 us from a store to its sight by the neighbour, more than
// the updates of a small brick, so the brick computes more to exchange less: its ring
// is two rows wide, and it updates the red cells of the first ring row itself, from the
// same values as their owner does (the same bits).  Only black values travel:
//     red, own rows and first ring row -> CTA barrier -> black, own rows
//     (published) -> black of both ring rows -> CTA barrier -> stop test.
// The black cells a red ring cell needs lie in the second ring row, in its own row and
// plane, and at the brick's corners, so a brick hears from its eight neighbours.  A
// published word goes to the inbox half of its sweep's parity: a neighbour may still
// read a sweep's words when the next sweep's arrive, but has read them before the
// ones after (it published those of the sweep between, which this CTA waited for).
//
// The stop rule (k_resident.cuh).  The verdicts of a sweep's two halves take longer to
// be summed over the CTAs than a sweep, so they are judged one sweep later: a solve that
// turns out to have ended a sweep ago takes e from before this sweep, which every update
// leaves beside the new value.  A cycle's last sweep is judged at once.  Restarts
// and the final p += e run in the kernel; d of the first ring row's red cells is kept
// and updated like the brick's own.  1/diag is formed from the coefficients.
// Rows of at most 32 cells per colour, two or more side by side on a warp's lanes.
//
// A sweep takes 2.6 us at 40^3 FP64 (3.4 with two hand-overs), 2.7 us at 61x47x53 FP32 (3.5),
// 2.75 us at 32x96x96 FP32 (3.8), 1.65 us at 12x10x8 FP64 (2.3, in one CTA).  Bound by the
// hand-over's trip (1.5 us) and, past some 40 rows a brick, by instruction issue: a turn of the 16
// warps over a row each takes 0.28 us FP32, 0.35 us FP64.  One row per warp and turn: with two, as
// the resident kernel takes them, half of a small brick's last turn is empty (32x96x96: 2.95 us).
// The verdicts judged in their own sweep: 3.0 us there.
#pragma once

#include "k_resident.cuh"

namespace ntcfd {

// Tile rows of a brick with its two ring rows; rows whose red cells it updates (bound).
__host__ __device__ inline int deep_tile_rows(const Brick& b) { return (b.JB + 4) * (b.KB + 4); }
__host__ __device__ inline int deep_red_rows(const Brick& b) { return (b.JB + 2) * (b.KB + 2); }
// Inbox rows: two per row of the faces j-low, j-high (KB long), k-low, k-high (JB), four corners.
__host__ __device__ inline int deep_inbox_rows(const Brick& b) { return 4 * (b.JB + b.KB) + 4; }

template <class Tc>
inline size_t deep_smem(const Brick& b) {
    // e, d and the sweep before's e of both colours, 64 words of slack (loads past the last row), then per red row its
    // coefficients and place, per own row its places in up to eight inboxes, the ring list
    return sizeof(Tc) * (6 * (size_t)deep_tile_rows(b) * b.mx + 64) + (size_t)deep_red_rows(b) * (4 * sizeof(Tc) + 8) +
           (size_t)b.JB * b.KB * 32 + (size_t)deep_inbox_rows(b) * 12 + 64;
}

template <class Tc, int NT>
__global__ void __launch_bounds__(NT, 1)
k_sor_deep(Geom g, SorCoef<Tc> sc, Brick br, double* __restrict__ p, const Tc* __restrict__ dRg,
           const Tc* __restrict__ dBg, Ctl* ctl, ResSync* sync, unsigned long long* boxes, double omega, double zeta,
           int itmax, int cycle_len, int check_every) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using B = decltype(abs_bits(Tc(0)));
    using Word = RingWord<Tc>;
    constexpr int NWARP = NT / 32, kFill = 24 / (int)sizeof(Tc);   // ring words a thread holds in flight
    __shared__ int s_flag, s_fail[2], s_nan[2];
    __shared__ uint2 s_vd;                        // this sweep's red verdicts, the last sweep's black ones
    __shared__ unsigned int s_prev[2][4];
    __shared__ int s_nr, s_ring;
    __shared__ B s_red_max[NWARP];
    const int JB = br.JB, KB = br.KB, mx = br.mx, RS = JB + 4, plane = RS * mx, tile = plane * (KB + 4);
    Tc* const S0 = reinterpret_cast<Tc*>(smem_raw);
    Tc* const S1 = S0 + tile;
    Tc* const D0 = S1 + tile;
    Tc* const D1 = D0 + tile;
    // per red row (own rows first): cN, cS, cF, cB; tile row start and (j+k)&1
    const int nrmax = deep_red_rows(br);
    Tc* const H0 = D1 + tile;                     // own cells' e before the last sweep
    Tc* const H1 = H0 + tile;
    auto align16 = [&](const void* q) { return smem_raw + (((size_t)((const unsigned char*)q - smem_raw) + 15) & ~size_t(15)); };
    Tc* const rowC = reinterpret_cast<Tc*>(align16(H1 + tile + 64));
    int2* const rowT = reinterpret_cast<int2*>(rowC + 4 * nrmax);
    int* const pubT = reinterpret_cast<int*>(align16(rowT + nrmax));      // words into the inboxes, eight per own row, -1: none
    int* const ringT = pubT + 8 * JB * KB;                       // inbox row, tile row start, (j+k)&1
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    const int bj = blockIdx.x % br.nbj, bk = blockIdx.x / br.nbj;
    const int j0 = 1 + brick_start(bj, g.ny, br.nbj), nj = 1 + brick_start(bj + 1, g.ny, br.nbj) - j0;
    const int k0 = 1 + brick_start(bk, g.nz, br.nbk), nk = 1 + brick_start(bk + 1, g.nz, br.nbk) - k0;
    const bool jlo = bj > 0, jhi = bj < br.nbj - 1, klo = bk > 0, khi = bk < br.nbk - 1;
    const int nown0 = g.nx / 2, nown1 = (g.nx + 1) / 2, nrows = nj * nk;
    auto place = [&](int jl, int kl) { return ((kl + 1) * RS + jl + 1) * mx; };   // jl, kl = -1 .. n + 2

    for (int q = tid; q < 6 * tile + 64; q += NT) S0[q] = Tc(0);
    if (tid == 0) {
        s_fail[0] = s_fail[1] = s_nan[0] = s_nan[1] = 0;
        s_vd = make_uint2(0u, 0u);
        s_nr = nrows;
        s_ring = 0;
    }
    if (tid < 8) s_prev[tid >> 2][tid & 3] = 0u;
    __syncthreads();
    auto red_row = [&](int slot, int jl, int kl) {
        const int j = j0 + jl - 1, k = k0 + kl - 1;
        rowT[slot] = make_int2(place(jl, kl), (j + k) & 1);
        rowC[4 * slot + 0] = sc.cN[j];
        rowC[4 * slot + 1] = sc.cS[j];
        rowC[4 * slot + 2] = sc.cF[k];
        rowC[4 * slot + 3] = sc.cB[k];
    };
    // own rows and where their black cells go
    const int rows_in = deep_inbox_rows(br);
    for (int er = tid; er < nrows; er += NT) {
        const int jl = er % nj + 1, kl = er / nj + 1;
        red_row(er, jl, kl);
        int n = 0;
        // the neighbour one brick along (dj, dk) keeps this row at `row` of its inbox (the first half's)
        auto to = [&](int dj, int dk, int row) {
            pubT[8 * er + n++] = (((int)blockIdx.x + dj + dk * br.nbj) * 2 * rows_in + row) * nown1 * Word::n;
        };
        if (jlo && jl <= 2) to(-1, 0, 2 * KB + (jl - 1) * KB + kl - 1);                  // its j-high face
        if (jhi && jl >= nj - 1) to(1, 0, (nj - jl) * KB + kl - 1);                      // its j-low face
        if (klo && kl <= 2) to(0, -1, 4 * KB + 2 * JB + (kl - 1) * JB + jl - 1);
        if (khi && kl >= nk - 1) to(0, 1, 4 * KB + (nk - kl) * JB + jl - 1);
        const int corner = 4 * (JB + KB);
        if (jlo && klo && jl == 1 && kl == 1) to(-1, -1, corner + 3);
        if (jhi && klo && jl == nj && kl == 1) to(1, -1, corner + 2);
        if (jlo && khi && jl == 1 && kl == nk) to(-1, 1, corner + 1);
        if (jhi && khi && jl == nj && kl == nk) to(1, 1, corner + 0);
        while (n < 8) pubT[8 * er + n++] = -1;
    }
    // the first ring row's red rows, and the rows that come from the inbox (black), in any order
    for (int q = tid; q < rows_in; q += NT) {
        int jl, kl, depth = 1;
        bool have;
        if (q < 4 * KB) {
            const int face = q / (2 * KB), d = q / KB & 1;
            kl = q % KB + 1;
            depth = d + 1;
            jl = face ? nj + depth : 1 - depth;
            have = kl <= nk && (face ? jhi : jlo);
        } else if (q < 4 * (JB + KB)) {
            const int r = q - 4 * KB, face = r / (2 * JB), d = r / JB & 1;
            jl = r % JB + 1;
            depth = d + 1;
            kl = face ? nk + depth : 1 - depth;
            have = jl <= nj && (face ? khi : klo);
        } else {
            const int c = q - 4 * (JB + KB);
            jl = c & 1 ? nj + 1 : 0;
            kl = c & 2 ? nk + 1 : 0;
            depth = 2;                                // no red of the corners
            have = (c & 1 ? jhi : jlo) && (c & 2 ? khi : klo);
        }
        if (!have) continue;
        const int at = atomicAdd(&s_ring, 1);
        ringT[3 * at] = q;
        ringT[3 * at + 1] = place(jl, kl);
        ringT[3 * at + 2] = (j0 + jl + k0 + kl) & 1;
        if (depth == 1) red_row(atomicAdd(&s_nr, 1), jl, kl);
    }
    __syncthreads();
    const int nr = s_nr, ring_tot = s_ring * nown1;
    // d: red of the red rows, black of the own ones
    for (int row = warp; row < nr; row += NWARP) {
        const int2 rt = rowT[row];
        const int kl = rt.x / plane - 1, jl = rt.x / mx % RS - 1;
        const long long gq = spl(g, 0, j0 + jl - 1, k0 + kl - 1);
        for (int m = lane; m < mx; m += 32) {
            D0[rt.x + m] = dRg[gq + m];
            if (row < nrows) D1[rt.x + m] = dBg[gq + m];
        }
    }
    const int rpw = 32 / nown1, sub = lane / nown1, lt = lane - sub * nown1;
    Tc cEr[2], cWr[2];                            // of the lane's cell in rows of parity 0, 1
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int i = min(2 * lt + 2 - r, g.nx + 2);
        cEr[r] = sc.cE[i];
        cWr[r] = sc.cW[i];
    }
    const unsigned int nblocks = gridDim.x, seq0 = sync->seq;
    const bool ctrl = tid == NT / 2;              // the thread that talks to the counters
    const int ik0 = ctl->ik;
    const Tc om = (Tc)omega;
    const size_t boxw = (size_t)rows_in * nown1 * Word::n;       // 8-byte words of an inbox half
    const unsigned int mH = 0xffffffffu / (unsigned)nown1 + 1u;  // q / nown1
    __syncthreads();

    // one colour over the first n rows, rpw rows per warp and turn; black is published under seq
    auto pass = [&](auto cc, int n, unsigned int seq, B& ch) {
        constexpr int c = decltype(cc)::value;
        Tc* const W = c ? S1 : S0;
        const Tc* const O = c ? S0 : S1;
        const Tc* const D = c ? D1 : D0;
        Tc* const H = c ? H1 : H0;
        unsigned long long* const box = boxes + (seq & 1u) * boxw + lt * Word::n;
        for (int er = rpw * warp + sub; er < n + sub; er += rpw * NWARP) {
            const bool in = sub < rpw && er < n;
            const int row = in ? er : 0;
            const int2 rt = rowT[row];
            const int r = (rt.y ^ c) & 1, m = rt.x + lt + 2 - r;
            const bool ok = in && lt < (r ? nown1 : nown0);
            const Tc* const o = O + m;
            Tc cN, cS, cF, cB;
            if constexpr (sizeof(Tc) == 4) {
                const float4 q = *reinterpret_cast<const float4*>(rowC + 4 * row);
                cN = q.x; cS = q.y; cF = q.z; cB = q.w;
            } else {
                const double2 q = *reinterpret_cast<const double2*>(rowC + 4 * row);
                const double2 t = *reinterpret_cast<const double2*>(rowC + 4 * row + 2);
                cN = q.x; cS = q.y; cF = t.x; cB = t.y;
            }
            const Tc cE = r ? cEr[1] : cEr[0], cW = r ? cWr[1] : cWr[0], e0 = W[m];
            const Tc rd = rdiag_near(((cE + cW) + (cN + cS)) + (cF + cB));
            Tc e1;
            const Tc diff = sor_update(cE, O[rt.x + lt + 2], cW, O[rt.x + lt + 1], cN, o[mx], cS, o[-mx], cF, o[plane], cB,
                                       o[-plane], rd, D[m], e0, om, &e1);
            if (ok) {
                W[m] = e1;
                H[m] = e0;
                if (c || row < nrows) {
                    const B b = abs_bits(diff);
                    ch = b > ch ? b : ch;
                }
            }
            if (c && in) {
                const Tc v = ok ? e1 : Tc(0);     // 0 where the row is a cell shorter than the ring
                const int4 ta = *reinterpret_cast<const int4*>(pubT + 8 * row);
                const int4 tb = *reinterpret_cast<const int4*>(pubT + 8 * row + 4);
                const int to[8] = {ta.x, ta.y, ta.z, ta.w, tb.x, tb.y, tb.z, tb.w};
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (to[q] >= 0) Word::store(box + to[q], v, seq);
            }
        }
    };
    using RedT = std::integral_constant<int, 0>;
    using BlackT = std::integral_constant<int, 1>;
    // the ring's black cells of seq, from this CTA's inbox; a CTA barrier follows
    auto fill = [&](unsigned int seq, int par) {
        const unsigned long long* const bx = boxes + ((size_t)blockIdx.x * 2 + (seq & 1u)) * boxw;
        for (int q0 = 0; q0 < ring_tot; q0 += NT * kFill) {
            Word w[kFill];
            const unsigned long long* at[kFill];
#pragma unroll
            for (int u = 0; u < kFill; ++u) {
                const int q = min(q0 + tid + NT * u, ring_tot - 1);
                const int r = (int)__umulhi((unsigned)q, mH);
                at[u] = bx + ((size_t)ringT[3 * r] * nown1 + (q - r * nown1)) * Word::n;
                w[u].load(at[u]);
            }
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
                for (int u = 0; u < kFill; ++u) w[u].load(at[u]);
            }
#pragma unroll
            for (int u = 0; u < kFill; ++u) {
                const int q = q0 + tid + NT * u;
                if (q >= ring_tot) continue;
                const int r = (int)__umulhi((unsigned)q, mH);
                // cell t of the row sits at m = t + 2 - parity
                S1[ringT[3 * r + 1] + (q - r * nown1) + 2 - (ringT[3 * r + 2] ^ 1)] = w[u].value();
            }
        }
    };
    // p += e of the own rows, a warp per row; with `defect` also d = the FP64 defect of
    // p + e (defect_update) of every cell whose d is kept
    // (undo: from e before the last sweep)
    auto correct = [&](bool defect, bool undo) {
        for (int q = warp; q < (defect ? nr : nrows); q += NWARP) {
            const int2 rt = rowT[q];
            const int kl = rt.x / plane - 1, jl = rt.x / mx % RS - 1, j = j0 + jl - 1, k = k0 + kl - 1;
            const bool own = q < nrows;
            const double cN = g.cN[j], cS = g.cS[j], cF = g.cF[k], cB = g.cB[k];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (c && !own) continue;
                const int r = (rt.y ^ c) & 1, m = rt.x + lane + 2 - r, i = 2 * lane + 2 - r;
                if (lane >= (r ? nown1 : nown0)) continue;
                const Tc e = undo ? (c ? H1 : H0)[m] : (c ? S1 : S0)[m];
                double* const pp = p + nat(g, i, j, k);
                const double pv = own ? *pp : 0.0;
                if (defect) {
                    const Tc* const O = c ? S0 : S1;
                    Tc* const D = c ? D1 : D0;
                    D[m] = (Tc)defect_update(g.cE[i], O[rt.x + lane + 2], g.cW[i], O[rt.x + lane + 1], cN, O[m + mx], cS,
                                             O[m - mx], cF, O[m + plane], cB, O[m - plane], D[m], e);
                }
                if (own) *pp = pv + (double)e;
            }
        }
    };
    const float zf = __double2float_rd(zeta);     // FP32 changes against the largest float <= zeta
    auto above = [&](B ch) {
        if constexpr (sizeof(Tc) == 4) return !(__uint_as_float(ch) <= zf);
        else return !(__longlong_as_double((long long)ch) <= zeta);
    };
    auto verdict = [&](int any, int par) {
        return 1ull | (unsigned long long)((any ? 1u : 0u) + (s_nan[par] ? kNanFlag : 0u)) << 32;
    };
    constexpr B kInf = sizeof(Tc) == 4 ? (B)0x7f800000u : (B)kInfBits;

    // The sums of sweep sg's verdicts to s_vd (red, black), once per sweep and in order; by
    // ctrl, from the counters as it saw them earlier (w).
    auto look = [&](int sg) {
        return make_ulonglong2(ld_relaxed(&sync->cnt[0][sg & 3]), ld_relaxed(&sync->cnt[1][sg & 3]));
    };
    auto judge = [&](int sg, int par, ulonglong2 w) {
        const unsigned int target = nblocks * (unsigned)((sg >> 2) + 1);
        const bool ok = ((int)((unsigned int)w.x - target) >= 0 ||
                         count_wait(&sync->cnt[0][sg & 3], target, &sync->bar.err, &w.x)) &&
                        ((int)((unsigned int)w.y - target) >= 0 ||
                         count_wait(&sync->cnt[1][sg & 3], target, &sync->bar.err, &w.y));
        if (!ok) s_fail[par] = 1;
        const unsigned int h0 = (unsigned int)(w.x >> 32), h1 = (unsigned int)(w.y >> 32);
        s_vd = make_uint2(h0 - s_prev[0][sg & 3], h1 - s_prev[1][sg & 3]);
        s_prev[0][sg & 3] = h0;
        s_prev[1][sg & 3] = h1;
    };
    int done = 0, done_c = 0, restarts = 0;
    bool conv = false, nonfinite = false, failed = false, tested = false, undo = false, added = false;
    B chs = B(0);
    double last = 0.0;
    for (;;) {
        done_c = 0;
        bool open = false, open_test = false;         // the sweep before is not judged yet; and is tested
#pragma unroll 1
        for (int s = 0; ik0 + done + s < itmax && s < cycle_len; ++s) {
            const int sg = done + s, par = sg & 1, ik = ik0 + sg + 1;
            const unsigned int seq = seq0 + (unsigned)sg + 1u;
            B cr = B(0), cb = B(0);
            pass(RedT{}, nr, seq, cr);
            if (cr >= kInf) s_nan[par] = 1;
            const int any_r = __syncthreads_or(above(cr));
            if (ctrl) red_add_relaxed(&sync->cnt[0][sg & 3], verdict(any_r, par));
            pass(BlackT{}, nrows, seq, cb);
            ulonglong2 w = make_ulonglong2(0ull, 0ull);
            if (ctrl && open) w = look(sg - 1);       // a trip through L2 ahead of its use
            fill(seq, par);
            if (ctrl && open) judge(sg - 1, par, w);
            if (cb >= kInf) s_nan[par] = 1;
            const int any_b = __syncthreads_or(above(cb));
            if (s_fail[par]) {
                failed = true;
                break;
            }
            if (ctrl) red_add_relaxed(&sync->cnt[1][sg & 3], verdict(any_b, par));
            if (open_test) {
                const uint2 vd = s_vd;
                nonfinite = vd.x >= kNanFlag || vd.y >= kNanFlag;
                conv = vd.x == 0u && vd.y == 0u;
                if (conv || nonfinite) {              // the solve ended with the sweep before
                    undo = true;
                    break;
                }
            }
            chs = cb > cr ? cb : cr;
            done_c = s + 1;
            open = true;
            open_test = check_every == 1 || ik >= itmax || ik % check_every == 0;
            tested = tested || open_test;
        }
        done += done_c;
        if (failed || undo) break;
        // another cycle only when this one ended on its length; its p += e and d do no harm to a
        // solve that turns out to have ended, and cover the judgement
        const bool again = done_c == cycle_len && ik0 + done < itmax;
        if (again) correct(true, false);
        added = again;
        if (open) {
            const int par = (done - 1) & 1;
            __syncthreads();                          // s_vd and s_fail have been read
            if (ctrl) judge(done - 1, par, look(done - 1));
            __syncthreads();
            if (s_fail[par]) {
                failed = true;
                break;
            }
            if (open_test) {
                nonfinite = s_vd.x >= kNanFlag || s_vd.y >= kNanFlag;
                conv = s_vd.x == 0u && s_vd.y == 0u;
            }
        }
        if (conv || nonfinite || !again) break;
        added = false;
        for (int q = tid; q < 2 * tile; q += NT) S0[q] = Tc(0);
        __syncthreads();
        ++restarts;
    }
    if (!added) correct(false, undo);
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
            atomicMax(&sync->last, widen_bits(b2));
        }
        GridPlace at;
        if (!grid_sync(&sync->bar, at, nblocks, &s_flag)) failed = true;
        else if (tid == 0) last = __longlong_as_double((long long)ld_relaxed(&sync->last));
    }
    if (blockIdx.x == 0 && tid == 0) {
        sync->seq = seq0 + (failed ? 1u << 24 : (unsigned)done + 8u);
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
