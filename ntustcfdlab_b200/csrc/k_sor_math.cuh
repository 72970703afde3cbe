// k_sor_math.cuh -- the arithmetic shared by every kernel of the pressure
// solve: the SOR update of a cell, the FP64 defect and its incremental form,
// all in explicitly rounded operations.
#pragma once

#include "ntcfd_common.cuh"

namespace ntcfd {

template <class Tc>
struct SorCoef {
    const Tc *cE, *cW, *cN, *cS, *cF, *cB;
};

__device__ __forceinline__ double rcp_rn(double x) { return __drcp_rn(x); }
__device__ __forceinline__ float rcp_rn(float x) { return __frcp_rn(x); }

// 1 / sum of the six coefficients (correctly rounded reciprocal)
template <class Tc>
__device__ __forceinline__ Tc rdiag_of(const SorCoef<Tc>& s, int i, int j, int k) {
    return rcp_rn(((s.cE[i] + s.cW[i]) + (s.cN[j] + s.cS[j])) + (s.cF[k] + s.cB[k]));
}

// Explicitly rounded operations: every kernel that evaluates a sweep or a
// defect uses these, so the resident and streaming paths round alike
// whatever the compiler would contract.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }

// One SOR update of a cell of the correction e (GS.f90:43-53 in the form
// eNew = rdiag * sum_nb c_nb e_nb + d): returns eNew - e0 and the relaxed
// value e0 + omega (eNew - e0) in *e1.
template <class Tc>
__device__ __forceinline__ Tc sor_update(Tc cE, Tc oE, Tc cW, Tc oW, Tc cN, Tc oN, Tc cS, Tc oS, Tc cF,
                                         Tc oF, Tc cB, Tc oB, Tc rd, Tc d, Tc e0, Tc om, Tc* e1) {
    Tc s = mul_rn(cE, oE);
    s = fma_rn(cW, oW, s);
    s = fma_rn(cN, oN, s);
    s = fma_rn(cS, oS, s);
    s = fma_rn(cF, oF, s);
    s = fma_rn(cB, oB, s);
    const Tc diff = sub_rn(fma_rn(rd, s, d), e0);
    *e1 = fma_rn(om, diff, e0);
    return diff;
}

// FP64 defect of a cell, d = rdiag * sum_nb c_nb p_nb - b' - p (the reference
// sweep's fixed-point residual), rd = rdiag_of of the cell: the same sums as
// sor_update.
__device__ __forceinline__ double defect_value(double cE, double pe, double cW, double pw, double cN, double pn,
                                               double cS, double ps, double cF, double pf, double cB, double pb,
                                               double rd, double bv, double pc) {
    double s = mul_rn(cE, pe);
    s = fma_rn(cW, pw, s);
    s = fma_rn(cN, pn, s);
    s = fma_rn(cS, ps, s);
    s = fma_rn(cF, pf, s);
    s = fma_rn(cB, pb, s);
    return sub_rn(fma_rn(rd, s, -bv), pc);
}

// FP64 reciprocal of a coefficient sum (positive and finite): the hardware's
// approximate double reciprocal refined by two Newton-Raphson steps
// x' = x + x (1 - s x), each of which squares the relative error.
__device__ __forceinline__ double rdiag64(double s) {
    double x;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(s));
    double r = fma_rn(-s, x, 1.0);
    x = fma_rn(x, r, x);
    r = fma_rn(-s, x, 1.0);
    x = fma_rn(x, r, x);
    return x;
}

// 1 / s to nearest, as rcp_rn gives it, for a normal sum with a normal reciprocal: the kernels that
// form 1/diag in a sweep take the same values as those that read it (make_rd).  The hardware's
// approximation, then steps whose remainder 1 - s x the FMA keeps exactly; the last one rounds to
// nearest when x is within an ulp (Markstein, IBM J. Res. Dev. 34, 1990).  FP32: one step (equal to
// rcp_rn for every significand).  FP64: a third-order step to within an ulp, rounded up, since the
// last step ties for a significand of ones only if it comes from below; then the last (equal for 10^11
// random sums, of which two Newton-Raphson steps miss 14 to 20).
__device__ __forceinline__ float rdiag_near(float s) {
    float x;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(x) : "f"(s));
    return fma_rn(x, fma_rn(-s, x, 1.0f), x);
}
__device__ __forceinline__ double rdiag_near(double s) {
    double x;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(s));
    const double r = fma_rn(-s, x, 1.0);
    x = __fma_ru(x, fma_rn(r, r, r), x);
    return fma_rn(x, fma_rn(-s, x, 1.0), x);
}

// The FP64 defect of p + e from the defect d of p and the correction e of a
// defect-correction cycle: since the operator is linear,
//     d' = rdiag sum c (p+e)_nb - b' - (p+e) = d + rdiag sum_nb c_nb e_nb - e,
// formed in FP64 with the FP64 coefficients from the cycle's (exact) Tc
// values of e; rdiag is rdiag64 of the FP64 coefficient sum.  Both SOR paths
// restart a cycle with it.
template <class Tc>
__device__ __forceinline__ double defect_update(double cE, Tc eE, double cW, Tc eW, double cN, Tc eN, double cS,
                                                Tc eS, double cF, Tc eF, double cB, Tc eB, Tc d, Tc e) {
    double s = mul_rn(cE, (double)eE);
    s = fma_rn(cW, (double)eW, s);
    s = fma_rn(cN, (double)eN, s);
    s = fma_rn(cS, (double)eS, s);
    s = fma_rn(cF, (double)eF, s);
    s = fma_rn(cB, (double)eB, s);
    const double x = rdiag64(((cE + cW) + (cN + cS)) + (cF + cB));
    return sub_rn(fma_rn(x, s, (double)d), (double)e);
}

}  // namespace ntcfd
