// Kernel functions K (value) and K' (first derivative factor) on prescaled
// coordinates, for the FP32 compensated path and the FP64 path.
//
// Reference: py-lddmm/kernelFunctions.f90 -- Gaussian (`ord > 4`):
//   K = exp(-u/2), K' = -exp(-u/2)/(2 s^2), u = |x-y|^2/s^2        (:33-40, :94-100)
// Laplacian of order p (0..4):
//   K = P_p(u) e^-u, K' = -Q_p(u) e^-u / (2 s^2), u = |x-y|/s          (:41-47, :101-107)
// with the polynomial tables c_ (P) and c1_ (Q).  Constant factors
// (-1/(2 s^2), the 2 of the gradient and the coordinate prescale) are applied
// once per target when its sums are written, not per pair.
//
// FP32 prescaling (done when points are packed):
//   Gaussian:  x' = x * sqrt(log2(e)/2)/s  ->  K  = 2^(-|x'-y'|^2)
//   Laplacian: x' = x * log2(e)/s          ->  u' = |x'-y'| = log2(e) u,
//              e^-u = 2^(-u'), polynomials rewritten in u' (c_j / log2(e)^j).
// The Fortran zero-distance branch (K = 1 when u < 1e-8) is a no-op in FP32:
// 2^(-t) for 0 <= t < 1.5e-8 rounds to 1.0f, and so does P(u)e^-u.
//
// FP64 sweeps: the same base-2 frame and exponential exp2neg below, with the
// zero-distance branch kept as in the Fortran.  FP64 sums that keep the
// reference's order to the bit (single-cluster kernels, sums over at most 384
// sources; LIB): x' = x/s, u = |x'-y'|^2 (Gaussian) or |x'-y'| (Laplacian)
// and exp() from the CUDA math library.
#pragma once
#include "common.cuh"

namespace lddmm {

// Polynomial in Horner form, DEG is the polynomial degree (coefficients c[0..DEG]).
template <int DEG>
LDDMM_D float horner(const float* c, float u) {
    float p = c[DEG];
#pragma unroll
    for (int j = DEG - 1; j >= 0; --j) p = fmaf(p, u, c[j]);
    return p;
}

// FP32 kernel value from the prescaled squared distance.
template <int KIND, int PDEG>
LDDMM_D float kval32(const float* pk, float r2) {
    if constexpr (KIND == KGAUSS) {
        return ex2(-r2);
    } else {
        const float u = sqrt_approx(r2);
        const float e = ex2(-u);
        if constexpr (PDEG == 0) return e;
        else return horner<PDEG>(pk, u) * e;
    }
}

// FP32 derivative factor: returns F with K'(x,y) 2 (x-y) = scale * F * (x'-y').
template <int KIND, int QDEG>
LDDMM_D float kdiff32(const float* pq, float r2) {
    if constexpr (KIND == KGAUSS) {
        return ex2(-r2);
    } else {
        const float u = sqrt_approx(r2);
        const float e = ex2(-u);
        if constexpr (QDEG == 0) return pq[0] * e;
        else return horner<QDEG>(pq, u) * e;
    }
}

// log2 of the kernel factor at a prescaled squared distance d2: K with its
// polynomial P, or the factor of K' with Q (both fall with the distance).  A
// few units of the last place are enough: it only bounds what far records add.
LDDMM_D float coef32(float c) { return c; }
LDDMM_D float coef32(double c) { return (float)c; }
LDDMM_D float coef32(unsigned long long dup) { return __uint_as_float((unsigned)dup); }
template <int KIND, int DEG, class C>
LDDMM_D float lg_factor(const C* c, float d2) {
    if constexpr (KIND == KGAUSS) {
        return -d2;
    } else {
        const float u = sqrt_approx(d2);
        float p = coef32(c[DEG]);
#pragma unroll
        for (int j = DEG - 1; j >= 0; --j) p = fmaf(p, u, coef32(c[j]));
        return __log2f(p) - u;
    }
}

// FP64 monomial-sum polynomial, evaluated like the Fortran expression
// c0 + c1*u + c2*u**2 + ... (left-to-right).
template <int DEG>
LDDMM_D double poly64(const double* c, double u) {
    double s = c[0];
    double up = 1.0;
#pragma unroll
    for (int j = 1; j <= DEG; ++j) {
        up = up * u;
        s = s + c[j] * up;
    }
    return s;
}

// 2^-x for x >= 0 in FP64, 0 from 2^-1022 on, NaN for NaN.
//
// x = k - f with k the nearest integer (adding and subtracting 1.5 2^52 rounds to
// it and leaves it in the low word), |f| <= 1/2, exact; 2^f = 1 + f q(f) with q of
// degree 10, the interpolant of (2^f - 1) / f at the 11 Chebyshev nodes of
// [-1/2, 1/2]: within 0.18 2^-53 of 2^f, 1.07 2^-53 with the rounding of the
// evaluation (2^f at 4000 points in 60 digits); 2^-k goes into the exponent.
//
// An FP64 pair was bound by issue slots, not by the FP64 pipe: about 64
// instructions, 26 of them FP64, most of them exp()'s range reduction, special
// cases and branches.  Here they are 3 additions and 11 fused multiply-adds plus
// eight integer instructions; the base-2 frame saves the multiplication by
// log2(e).  B200, n = m = 32,768: Gaussian applyK 4.5 -> 6.5, varifold value 4.0 ->
// 5.7, varifold gradient 3.4 -> 4.2, adjoint 3.7 -> 4.9 (1e11 pairs/s); the FP64 pipe
// (1.86e13 instructions/s, 23 of them per applyK pair) allows 8.1.
LDDMM_D double exp2neg(double x) {
    const double magic = 6755399441055744.0;
    const double t = __dadd_rn(x, magic);
    const double f = __dsub_rn(__dsub_rn(t, magic), x);
    double p = 0x1.e9d3fe3952179p-32;
    p = __fma_rn(p, f, 0x1.e6063f7217bc6p-28);
    p = __fma_rn(p, f, 0x1.b524fae627834p-24);
    p = __fma_rn(p, f, 0x1.62bfd47773353p-20);
    p = __fma_rn(p, f, 0x1.ffcbfc670dcd4p-17);
    p = __fma_rn(p, f, 0x1.430913096fd9fp-13);
    p = __fma_rn(p, f, 0x1.5d87fe78a5276p-10);
    p = __fma_rn(p, f, 0x1.3b2ab6fba1ddap-7);
    p = __fma_rn(p, f, 0x1.c6b08d704a0c2p-5);
    p = __fma_rn(p, f, 0x1.ebfbdff82c598p-3);
    p = __fma_rn(p, f, 0x1.62e42fefa39efp-1);
    p = __fma_rn(p, f, 1.0);
    const unsigned hx = (unsigned)__double2hiint(x);
    const bool big = hx >= 0x408FF000u;   // x >= 1022, or NaN
    const int hi = __double2hiint(p) - (__double2loint(t) << 20);
    return __hiloint2double(big ? (hx > 0x7FF00000u ? (int)hx : 0) : hi, big ? 0 : __double2loint(p));
}

// a < b for a >= 0 or NaN and b > 0, compared as integers (the FP64 pipe is the scarce
// one).  Unsigned, so that a NaN of either sign is not below b: inf - inf has its sign
// bit set, and as a signed integer it would be.
LDDMM_D bool less_nonneg(double a, double b) {
    return (unsigned long long)__double_as_longlong(a) < (unsigned long long)__double_as_longlong(b);
}

// the zero-distance thresholds in the base-2 frame
static constexpr double kLog2e = 1.4426950408889634;
static constexpr double kZero2Gauss = kZeroThresh * 0.5 * kLog2e;
static constexpr double kZero2Lap = kZeroThresh * kLog2e;

template <int KIND, int PDEG, bool LIB>
LDDMM_D double kval64(const double* pk, double r2) {
    if constexpr (LIB) {
        if constexpr (KIND == KGAUSS) {
            if (r2 < kZeroThresh) return 1.0;
            return exp(-0.5 * r2);
        } else {
            const double u = sqrt(r2);
            if (u < kZeroThresh) return 1.0;
            return poly64<PDEG>(pk, u) * exp(-1.0 * u);
        }
    } else if constexpr (KIND == KGAUSS) {
        const double e = exp2neg(r2);
        return less_nonneg(r2, kZero2Gauss) ? 1.0 : e;
    } else {
        const double u = sqrt(r2);
        const double k = poly64<PDEG>(pk, u) * exp2neg(u);
        return less_nonneg(u, kZero2Lap) ? 1.0 : k;
    }
}

template <int KIND, int QDEG, bool LIB>
LDDMM_D double kdiff64(const double* pq, double r2) {
    if constexpr (KIND == KGAUSS) {
        return kval64<KIND, 0, LIB>(pq, r2);
    } else if constexpr (LIB) {
        const double u = sqrt(r2);
        if (u < kZeroThresh) return pq[0];
        return poly64<QDEG>(pq, u) * exp(-1.0 * u);
    } else {
        const double u = sqrt(r2);
        const double k = poly64<QDEG>(pq, u) * exp2neg(u);
        return less_nonneg(u, kZero2Lap) ? pq[0] : k;
    }
}

}  // namespace lddmm
