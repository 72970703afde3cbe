// k_mask.cuh -- K7 immersed-boundary volume fraction ETA.
//
// K7 follows RayCasting (airfoil.f90:580-915): even-odd ray crossings per
// (k,j) cell centre against the polygon edges (ray towards +z), then 50x50
// sub-cells on the cells that hold a polygon vertex, then extrusion along
// i.  The reference moves the grid by 0.01 when a vertex ties exactly with
// a node coordinate (airfoil.f90:700-702,731-733,804-807,834-837); the
// device kernels count such ties instead and the host rejects the mask.
// K7b follows DFIB_Cylinder (DFIB.f90:74-145) in real*4 arithmetic.
#pragma once

#include "ntcfd_common.cuh"

namespace ntcfd {

// A list of polygon edges in shared memory, filled by the block NT edges at a time.
template <int NT>
struct EdgeList {
    double a0[NT], a1[NT], z0[NT], z1[NT];           // ay, az of the edge's ends
    int count[2];                                    // listed of this pass, and of the next
    // Lists the edges m0 .. m0 + NT - 1 that `keep` takes; every thread of the block.
    template <class Keep>
    __device__ __forceinline__ int fill(int m0, int pass, const double* az, const double* ay, int poly, Keep&& keep) {
        const int m = m0 + threadIdx.x;
        if (m < poly - 1) {
            const double p0 = ay[m], p1 = ay[m + 1], q0 = az[m], q1 = az[m + 1];
            if (keep(p0, p1, q0, q1)) {
                const int e = atomicAdd(&count[pass], 1);
                a0[e] = p0; a1[e] = p1; z0[e] = q0; z1[e] = q1;
            }
        }
        if (threadIdx.x == 0) count[pass ^ 1] = 0;
        __syncthreads();
        return count[pass];
    }
};

// ETA_1 of the cells k of row j from their crossing parity (airfoil.f90:685-764), a thread
// per cell.  Y, Z: node coordinates pre-offset (Y[j] valid for j in -1..n+3).
//
// Only edges that span the row's cell centres count, so the block lists those (some 2 to 30 of
// 511 for an airfoil) and its threads test the list: 64x192x256 6 us against
// 73 us with every cell testing every edge from memory.
template <int NT>
__device__ __forceinline__ void ray_main_row(int k, int j, int nz, const double* Y, const double* Z,
                                             const double* az, const double* ay, int poly, double* eta1,
                                             int* ties, EdgeList<NT>& ed) {
    const double Yj = Y[j], ycell = (Y[j] + Y[j + 1]) / 2.0;
    const bool in = k <= nz;
    const double Zk = in ? Z[k] : 0.0, zcell = in ? (Z[k] + Z[k + 1]) / 2.0 : 0.0;
    int cnt = 0, tie = 0;
    if (threadIdx.x == 0) ed.count[0] = 0;
    __syncthreads();
    for (int m0 = 0, pass = 0; m0 < poly - 1; m0 += NT, pass ^= 1) {
        const int count = ed.fill(m0, pass, az, ay, poly, [&](double a0, double a1, double, double) {
            return (a0 >= ycell && a1 <= ycell) || (a0 <= ycell && a1 >= ycell);
        });
        for (int e = 0; in && e < count; ++e) {
            const double a0 = ed.a0[e], a1 = ed.a1[e], z0 = ed.z0[e], z1 = ed.z1[e];
            const bool down = a0 >= ycell && a1 <= ycell, up = a0 <= ycell && a1 >= ycell;
            if (zcell >= fmax(z0, z1)) continue;
            if (zcell < fmin(z0, z1)) {
                cnt += (down ? 1 : 0) + (up ? 1 : 0);
                continue;
            }
            if (down) {
                if (Yj == a1 || Zk == z1) ++tie;
                if ((Yj - a1) / (Zk - z1) > (a0 - a1) / (z0 - z1)) ++cnt;
            }
            if (up) {
                if (Yj == a0 || Zk == z0) ++tie;
                if ((Yj - a0) / (Zk - z0) > (a1 - a0) / (z1 - z0)) ++cnt;
            }
        }
        __syncthreads();                             // the list is read
    }
    if (in) eta1[(long long)(k - 1) + (long long)nz * (j - 1)] = (cnt % 2 == 0) ? 0.0 : 1.0;
    if (tie) atomicAdd(ties, tie);
}

// The cell that holds polygon vertex m, in [Z(k),Z(k+1)) x [Y(j),Y(j+1)) for k in C..E-1, j in
// A..B-1 (airfoil.f90:661-674): flagged and, by the first vertex found in it, listed.  One
// warp per vertex (a thread per vertex walks the nodes one load after another: 34 us
// for 512 vertices on 192x256 nodes, 6 us by warps).
__device__ __forceinline__ void ray_point(int m, int ny, int nz, const double* Y, const double* Z,
                                          const double* az, const double* ay, int A, int B, int C, int E,
                                          int* flags, int* list, int* count) {
    const int lane = threadIdx.x & 31;
    const double z = az[m], y = ay[m];
    for (int k0 = C; k0 <= E - 1; k0 += 32) {
        const int kl = k0 + lane;
        unsigned int hit = __ballot_sync(0xffffffffu, kl <= E - 1 && z >= Z[kl] && z < Z[kl + 1]);
        for (; hit; hit &= hit - 1) {
            const int k = k0 + __ffs(hit) - 1;
            for (int j = A + lane; j <= B - 1; j += 32)
                if (y >= Y[j] && y < Y[j + 1] && k >= 1 && k <= nz && j >= 1 && j <= ny) {
                    const int q = (k - 1) + nz * (j - 1);
                    if (atomicExch(&flags[q], 1) == 0) list[atomicAdd(count, 1)] = q;
                }
        }
    }
}

// Sub-grid volume fraction of cut cell `cell` (airfoil.f90:773-884): the
// block's threads share the 50 x 50 sub-cells, ETA_1 = odd sub-cells / 2500.
//
// A sub-cell's ray meets only edges that span its y and do not lie wholly before its z.  The
// block lists the edges that span some y of the cell and end at or beyond its Z(k); a warp
// takes a row of sub-cells, finds the listed edges that span the row, a lane each, and
// tests those for its 50 sub-cells.  The edges left out change no count and no tie.
// 64x192x256 with 511 edges (an airfoil of chord 1): 15 us against 475 us with every edge
// tested for every sub-cell.
constexpr int kSub = 50;
template <int NT>
struct RaySub {
    double YY[kSub + 1], ZZ[kSub + 1];               // sub-cell nodes
    EdgeList<NT> ed;
    int odd[NT / 32];
};
template <int NT>
__device__ __forceinline__ void ray_sub_cell(int cell, int nz, const double* Y, const double* Z, const double* az,
                                             const double* ay, int poly, double* eta1, int* ties, RaySub<NT>& sm) {
    constexpr int kW = NT / 32, kRows = (kSub + kW - 1) / kW;   // warps, rows of a warp
    static_assert(kSub <= 64 && 2 * kRows <= 32 && NT > kSub, "two sub-cells of a row per lane, a bit each");
    const int k = cell % nz + 1, j = cell / nz + 1, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const double Yj = Y[j], Yj1 = Y[j + 1], Zk = Z[k], Zk1 = Z[k + 1];
    if (t <= kSub) {
        sm.YY[t] = Yj + t * (Yj1 - Yj) / (double)kSub;
        sm.ZZ[t] = Zk + t * (Zk1 - Zk) / (double)kSub;
    }
    if (t == 0) sm.ed.count[0] = 0;
    __syncthreads();
    unsigned int par = 0u;                           // parity of the lane's sub-cells: rows' pairs of bits
    int tie = 0;
    const EdgeList<NT>& ed = sm.ed;
    for (int m0 = 0, pass = 0; m0 < poly - 1; m0 += NT, pass ^= 1) {
        const int count = sm.ed.fill(m0, pass, az, ay, poly, [&](double a0, double a1, double z0, double z1) {
            return fmax(a0, a1) >= fmin(Yj, Yj1) && fmin(a0, a1) <= fmax(Yj, Yj1) && !(fmax(z0, z1) < fmin(Zk, Zk1));
        });
        for (int i = 0; i < kRows; ++i) {
            const int l = warp + i * kW;             // sub_intersection(.,l+1)
            if (l >= kSub) break;
            const double YYl = sm.YY[l], ycell = (YYl + sm.YY[l + 1]) / 2.0;
            for (int e0 = 0; e0 < count; e0 += 32) {
                const int el = e0 + lane;
                const bool ok = el < count;
                const double s0 = ok ? ed.a0[el] : 0.0, s1 = ok ? ed.a1[el] : 0.0;
                unsigned int downs = __ballot_sync(0xffffffffu, ok && s0 >= ycell && s1 <= ycell);
                unsigned int ups = __ballot_sync(0xffffffffu, ok && s0 <= ycell && s1 >= ycell);
                for (unsigned int hit = downs | ups; hit; hit &= hit - 1) {
                    const int b = __ffs(hit) - 1, e = e0 + b;
                    const bool down = (downs >> b) & 1u, up = (ups >> b) & 1u;
                    const double a0 = ed.a0[e], a1 = ed.a1[e], z0 = ed.z0[e], z1 = ed.z1[e];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int n = lane + 32 * h;     // sub_intersection(n+1,.)
                        if (n >= kSub) continue;
                        const double ZZn = sm.ZZ[n], zcell = (ZZn + sm.ZZ[n + 1]) / 2.0;
                        if (zcell > fmax(z0, z1)) continue;
                        int cnt = 0;
                        if (zcell < fmin(z0, z1)) cnt = (down ? 1 : 0) + (up ? 1 : 0);
                        else {
                            const bool at = YYl == a1 || ZZn == z1;
                            if (down) {
                                tie += at;
                                if ((YYl - a1) / (ZZn - z1) > (a0 - a1) / (z0 - z1)) ++cnt;
                            }
                            if (up) {
                                tie += at;
                                if ((YYl - a0) / (ZZn - z0) > (a1 - a0) / (z1 - z0)) ++cnt;
                            }
                        }
                        par ^= (unsigned int)(cnt & 1) << (2 * i + h);
                    }
                }
            }
        }
        __syncthreads();                             // the list is read
    }
    const int odd = __reduce_add_sync(0xffffffffu, __popc(par));
    if (lane == 0) sm.odd[warp] = odd;
    __syncthreads();
    if (t == 0) {
        int all = 0;
        for (int w = 0; w < kW; ++w) all += sm.odd[w];
        eta1[(long long)(k - 1) + (long long)nz * (j - 1)] = (double)all / (double)kSub / (double)kSub;
    }
    if (tie) atomicAdd(ties, tie);
    __syncthreads();                                 // the block's next cell
}

// ETA(i,j,k) = ETA_1(k,j) on the interior (airfoil.f90:889-891); ghosts 0.
__global__ void k_extrude(Geom g, const double* eta1, double* eta) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x - 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y - 1;
    const int k = blockIdx.z * blockDim.z + threadIdx.z - 1;
    if (i > g.nx + 2 || j > g.ny + 2 || k > g.nz + 2) return;
    const bool in = i >= 1 && i <= g.nx && j >= 1 && j <= g.ny && k >= 1 && k <= g.nz;
    eta[nat(g, i, j, k)] = in ? eta1[(long long)(k - 1) + (long long)g.nz * (j - 1)] : 0.0;
}

// ---- A smoothed, differentiable mask (no counterpart in the reference): the
// polygon moved as the ray cast moves it, ETA_1 a C1 ramp of the signed
// distance d from the (y,z) cell centre to the polygon (negative inside):
//     tau = -d / width,  ETA_1 = 1 (tau >= 1), 0 (tau <= -1),
//     0.5 + 0.75 tau - 0.25 tau^3 between,
// and dETA_1/dalpha from the vertices' derivatives (dpz, dpy) with respect to
// the angle: d is the distance to the nearest point Q = A + t (B - A) of the
// nearest edge, so dd/dalpha = -s n.((1 - t) dA + t dB), n the unit vector
// from Q to the centre, s = -1 inside.  Inside/outside by crossing parity.
__global__ void k_smooth_mask(int ny, int nz, const double* Y, const double* Z, const double* pz,
                              const double* py, const double* dpz, const double* dpy, int npts, double width,
                              double* eta1, double* deta1) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    if (k > nz || j > ny) return;
    const double yc = (Y[j] + Y[j + 1]) / 2.0, zc = (Z[k] + Z[k + 1]) / 2.0;
    double best = INFINITY, bt = 0.0;
    int bm = 0;
    bool inside = false;
    for (int m = 0; m < npts - 1; ++m) {
        const double az = pz[m], ay = py[m], bz = pz[m + 1], by = py[m + 1];
        const double abz = bz - az, aby = by - ay, apz = zc - az, apy = yc - ay;
        const double l2 = abz * abz + aby * aby;
        const double t = l2 > 0.0 ? fmin(fmax((apz * abz + apy * aby) / l2, 0.0), 1.0) : 0.0;
        const double qz = zc - (az + t * abz), qy = yc - (ay + t * aby);
        const double d2 = qz * qz + qy * qy;
        if (d2 < best) { best = d2; bt = t; bm = m; }
        if ((ay > yc) != (by > yc)) {
            const double zi = az + (yc - ay) * abz / aby;
            if (zc < zi) inside = !inside;
        }
    }
    const double du = sqrt(best), sgn = inside ? -1.0 : 1.0;
    const double tau = -sgn * du / width;
    double e, de = 0.0;
    if (tau >= 1.0) e = 1.0;
    else if (tau <= -1.0) e = 0.0;
    else {
        e = 0.5 + 0.75 * tau - 0.25 * tau * tau * tau;
        if (du > 0.0) {
            const double az = pz[bm], ay = py[bm];
            const double qz = az + bt * (pz[bm + 1] - az), qy = ay + bt * (py[bm + 1] - ay);
            const double nz_ = (zc - qz) / du, ny_ = (yc - qy) / du;
            const double dqz = (1.0 - bt) * dpz[bm] + bt * dpz[bm + 1];
            const double dqy = (1.0 - bt) * dpy[bm] + bt * dpy[bm + 1];
            const double ddu = -(nz_ * dqz + ny_ * dqy);
            de = 0.75 * (1.0 - tau * tau) * (-sgn * ddu / width);
        }
    }
    const long long q = (long long)(k - 1) + (long long)nz * (j - 1);
    eta1[q] = e;
    deta1[q] = de;
}

// ---- The ray cast on the device: a body set by the host, or the mask of a moving
// body, one step at a time inside the step graph (ntcfd_set_dynamic_aoa).  The host evaluates each step's angle
// (airfoil.f90:313-317) and its cosine and sine; k_dyn_rotate turns the body
// polygon by them (airfoil.f90:597-611) for the step the control block's step
// counter names.  After a step whose polygon meets an exact vertex/grid tie (the
// reference moves the grid instead) the control block's halt flag is set: the
// mask kernels and, through the graph's IF node, the step itself do nothing
// for the rest of the call.
struct DynMask {
    const double* base;   // body polygon: az[npts], then ay[npts]
    const double* trig;   // cos, sin of each step of the call
    double* poly;         // this step's polygon: az, then ay
    int npts;
    double zc, yc;
    int* flags;           // ny*nz: cells that hold a vertex (k fastest)
    int* list;            // ny*nz: those cells, compacted
    int* meta;            // A, B, C, E (airfoil.f90:615-654), listed cells, ties
    double* eta1;         // ETA_1(k,j)
};

// The step's polygon and its bounds A, B, C, E (airfoil.f90:615-654: A = the
// first j with Y(j) > min ay, less one, 0 when there is none; B = the first j
// with Y(j) > max ay; C, E likewise in z); the counters cleared.  One block.
// The rotation keeps the reference's order of operations (the new az enters
// the new ay) with every product and sum rounded on its own, as on the host.
template <int NT>
__global__ void __launch_bounds__(NT) k_dyn_rotate(int ny, int nz, const double* Y, const double* Z, DynMask m,
                                                   const Ctl* ctl) {
    if (ctl->halt) return;
    __shared__ double sd[4][NT];
    __shared__ int si[4][NT];
    const double c = m.trig[2 * ctl->step], sn = m.trig[2 * ctl->step + 1];
    const int t = threadIdx.x;
    double mny = INFINITY, mxy = -INFINITY, mnz = INFINITY, mxz = -INFINITY;
    for (int q = t; q < m.npts; q += NT) {
        const double z0 = __dsub_rn(m.base[q], 0.25), y0 = m.base[m.npts + q];
        const double z1 = __dsub_rn(__dmul_rn(c, z0), __dmul_rn(sn, y0));
        const double y1 = __dadd_rn(__dmul_rn(sn, z1), __dmul_rn(c, y0));
        const double az = __dadd_rn(__dadd_rn(z1, m.zc), 0.25), ay = __dadd_rn(y1, m.yc);
        m.poly[q] = az;
        m.poly[m.npts + q] = ay;
        mny = fmin(mny, ay); mxy = fmax(mxy, ay);
        mnz = fmin(mnz, az); mxz = fmax(mxz, az);
    }
    sd[0][t] = mny; sd[1][t] = mxy; sd[2][t] = mnz; sd[3][t] = mxz;
    __syncthreads();
    for (int s = NT / 2; s > 0; s >>= 1) {
        if (t < s) {
            sd[0][t] = fmin(sd[0][t], sd[0][t + s]); sd[1][t] = fmax(sd[1][t], sd[1][t + s]);
            sd[2][t] = fmin(sd[2][t], sd[2][t + s]); sd[3][t] = fmax(sd[3][t], sd[3][t + s]);
        }
        __syncthreads();
    }
    mny = sd[0][0]; mxy = sd[1][0]; mnz = sd[2][0]; mxz = sd[3][0];
    const int none = 0x7fffffff;
    int fa = none, fb = none, fc = none, fe = none;
    for (int j = t + 1; j <= ny; j += NT) {
        if (Y[j] > mny) fa = min(fa, j);
        if (Y[j] > mxy) fb = min(fb, j);
    }
    for (int k = t + 1; k <= nz; k += NT) {
        if (Z[k] > mnz) fc = min(fc, k);
        if (Z[k] > mxz) fe = min(fe, k);
    }
    si[0][t] = fa; si[1][t] = fb; si[2][t] = fc; si[3][t] = fe;
    __syncthreads();
    for (int s = NT / 2; s > 0; s >>= 1) {
        if (t < s)
            for (int q = 0; q < 4; ++q) si[q][t] = min(si[q][t], si[q][t + s]);
        __syncthreads();
    }
    if (t == 0) {
        m.meta[0] = si[0][0] == none ? 0 : si[0][0] - 1;
        m.meta[1] = si[1][0] == none ? 0 : si[1][0];
        m.meta[2] = si[2][0] == none ? 0 : si[2][0] - 1;
        m.meta[3] = si[3][0] == none ? 0 : si[3][0];
        m.meta[4] = 0;
        m.meta[5] = 0;
    }
}

// Crossing parity of every (k,j) cell, a block per part of a row j; the cut-cell flags cleared.
template <int NT>
__global__ void __launch_bounds__(NT) k_dyn_main(int ny, int nz, const double* Y, const double* Z, DynMask m,
                                                 const Ctl* ctl) {
    if (ctl->halt) return;
    __shared__ EdgeList<NT> ed;
    const double* az = m.poly;
    for (int j = blockIdx.y + 1; j <= ny; j += gridDim.y) {
        const int k = blockIdx.x * NT + threadIdx.x + 1;
        if (k <= nz) m.flags[(long long)(k - 1) + (long long)nz * (j - 1)] = 0;
        ray_main_row<NT>(k, j, nz, Y, Z, az, az + m.npts, m.npts, m.eta1, &m.meta[5], ed);
    }
}

// The cells that hold a vertex (within the bounds), flagged and listed (in any order: each
// is computed on its own).
__global__ void k_dyn_points(int ny, int nz, const double* Y, const double* Z, DynMask m, const Ctl* ctl) {
    if (ctl->halt) return;
    const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (q >= m.npts) return;
    const double* az = m.poly;
    ray_point(q, ny, nz, Y, Z, az, az + m.npts, m.meta[0], m.meta[1], m.meta[2], m.meta[3], m.flags, m.list,
              &m.meta[4]);
}

// Sub-cell fractions of the listed cells; blocks stride over the list.
template <int NT>
__global__ void __launch_bounds__(NT) k_dyn_sub(int nz, const double* Y, const double* Z, DynMask m,
                                                const Ctl* ctl) {
    if (ctl->halt) return;
    __shared__ RaySub<NT> sm;
    const double* az = m.poly;
    const int count = m.meta[4];
    for (int q = blockIdx.x; q < count; q += gridDim.x)
        ray_sub_cell<NT>(m.list[q], nz, Y, Z, az, az + m.npts, m.npts, m.eta1, &m.meta[5], sm);
}

// ETA from ETA_1, as k_extrude.
__global__ void k_dyn_extrude(Geom g, const double* eta1, double* eta, const Ctl* ctl) {
    if (ctl->halt) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x - 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y - 1;
    const int k = blockIdx.z * blockDim.z + threadIdx.z - 1;
    if (i > g.nx + 2 || j > g.ny + 2 || k > g.nz + 2) return;
    const bool in = i >= 1 && i <= g.nx && j >= 1 && j <= g.ny && k >= 1 && k <= g.nz;
    eta[nat(g, i, j, k)] = in ? eta1[(long long)(k - 1) + (long long)g.nz * (j - 1)] : 0.0;
}

// The step runs (IF condition 1) unless this or an earlier step of the call met
// a tie; the first such step's tie count is kept in the control block.
__global__ void k_dyn_gate(DynMask m, Ctl* ctl, cudaGraphConditionalHandle h) {
    if (!ctl->halt && m.meta[5] > 0) {
        ctl->halt = 1;
        ctl->halt_ties = m.meta[5];
    }
    cudaGraphSetConditional(h, ctl->halt ? 0u : 1u);
}

// DFIB_Cylinder (DFIB.f90:90-131): axis along x, centre (zc, yc), radius r.
// DISTANCE, DIAGONAL, SZ, SY, xi are real*4 as declared in DFIB.f90:78-85.
__global__ void k_cylinder(int ny, int nz, const double* Y, const double* Z, const double* iDx,
                           const double* iDy, const double* iDz, double zc, double yc, double r,
                           double* eta1) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    if (k > nz || j > ny) return;
    const int i = 1;
    // explicit _rn products and sums: no contraction into FMA, as in the
    // reference's separately rounded operations
    const float DIAGONAL = __double2float_rn(
        sqrt(__dadd_rn(__dadd_rn(__dmul_rn(iDx[i], iDx[i]), __dmul_rn(iDy[j], iDy[j])),
                       __dmul_rn(iDz[k], iDz[k]))) / 2.0);
    const double dzc = ((Z[k] + Z[k + 1]) / 2.0) - zc;
    const double dyc = ((Y[j] + Y[j + 1]) / 2.0) - yc;
    const float DISTANCE = __double2float_rn(sqrt(__dadd_rn(__dmul_rn(dzc, dzc), __dmul_rn(dyc, dyc))));
    double eta;
    if (fabs((double)DISTANCE - r) < (double)DIAGONAL) {
        float xi = 0.0f;
        const float dzg = __double2float_rn(iDz[k] / kSub);
        const float dyg = __double2float_rn(iDy[j] / kSub);
        for (int m = 1; m <= kSub; ++m) {
            const float SYm = __double2float_rn(Y[j] + (double)__fmul_rn((float)(m - 1), dyg));
            const float SYm1 = __double2float_rn(Y[j] + (double)__fmul_rn((float)(m), dyg));
            const double sy = (double)__fadd_rn(SYm, SYm1) / 2.0 - yc;
            for (int n = 1; n <= kSub; ++n) {
                const float SZn = __double2float_rn(Z[k] + (double)__fmul_rn((float)(n - 1), dzg));
                const float SZn1 = __double2float_rn(Z[k] + (double)__fmul_rn((float)(n), dzg));
                const double sz = (double)__fadd_rn(SZn, SZn1) / 2.0 - zc;
                const float SDIST = __double2float_rn(sqrt(__dadd_rn(__dmul_rn(sz, sz), __dmul_rn(sy, sy))));
                if ((double)SDIST <= r) xi = __fadd_rn(xi, 1.0f);
            }
        }
        eta = (double)__fdiv_rn(xi, (float)(kSub * kSub));
    } else if ((double)DISTANCE > r) {
        eta = 0.0;
    } else {
        eta = 1.0;
    }
    eta1[(long long)(k - 1) + (long long)nz * (j - 1)] = eta;
}

}  // namespace ntcfd
