// Pair operators plugged into sweep_kernel (sweep.cuh).
//
//   OpApplyK<Real, KIND, DEG, D, DIMB>   f_k = sum_l K(x_k,y_l) beta_l
//       py-lddmm/kernelFunctions.f90:1-54 (applyk)
//   OpDiffKT<Real, KIND, DEG, D, W>      f_k = sum_l K'(x_k,y_l) 2(x_k-y_l) <u_k, v_l>
//       py-lddmm/kernelFunctions.f90:56-114 (applykdifft), with
//       u_k = a1[:,k,:], v_l = a2[:,l,:] flattened to W = na*dimb entries.
//
// Packed layouts (all planes are arrays of 16-byte words, one word per record):
//   FP32 points : plane 0 = (x', y', z', 0) float4
//   FP32 weights: plane 1.. = 4 floats per plane
//   FP64 points : planes 0,1 = (x', y') (z', 0) double2 words
//   FP64 weights: 2 doubles per plane
#pragma once
#include "kfun.cuh"
#include "sweep.cuh"

namespace lddmm {

template <class Real>
struct AccFor;
template <>
struct AccFor<float> {
    template <int N>
    using type = AccF32C<N>;
};
template <>
struct AccFor<double> {
    template <int N>
    using type = AccF64<N>;
};

// LIB (FP64): exp() of the CUDA library in the x/s frame, see kfun.cuh
template <class Real, int KIND, int DEG, bool LIB>
LDDMM_D Real kval(const Real* pk, Real r2) {
    if constexpr (sizeof(Real) == 4) return kval32<KIND, DEG>(pk, r2);
    else return kval64<KIND, DEG, LIB>(pk, r2);
}
template <class Real, int KIND, int DEG, bool LIB>
LDDMM_D Real kdiff(const Real* pq, Real r2) {
    if constexpr (sizeof(Real) == 4) return kdiff32<KIND, DEG>(pq, r2);
    else return kdiff64<KIND, DEG, LIB>(pq, r2);
}

template <class Real>
struct KernelParamsBase {
    const float4* src4;      // source planes
    long long src_stride;    // words per source plane
    const float4* tgt4;      // target planes
    long long tgt_stride;    // words per target plane
    Real pk[5];              // K polynomial (prescaled), Laplacian only
    Real pq[4];              // K' polynomial (prescaled), Laplacian only
};

// Point planes per record: FP32 one float4, FP64 two double2 words.
template <class Real>
struct PointPlanes {
    static constexpr int N = (sizeof(Real) == 4) ? 1 : 2;
};

// ---------------------------------------------------------------------------
// f_k = sum_l K(x_k, y_l) beta_l
// ---------------------------------------------------------------------------
// SMALL: two targets per thread instead of four, for a few thousand targets or fewer
template <class Real_, int KIND, int DEG, int D, int DIMB, bool SMALL = false>
struct OpApplyK {
    using Real = Real_;
    static constexpr bool F32 = sizeof(Real) == 4;
    static constexpr int FAMILY = KIND;
    static constexpr int TPS = 1;
    static constexpr int R = (F32 && !SMALL) ? 4 : 2;
    static constexpr int PP = PointPlanes<Real>::N;
    static constexpr int WP = (DIMB + Traits<Real>::PER_WORD - 1) / Traits<Real>::PER_WORD;
    static constexpr int NS = PP + WP;
    static constexpr int NOUT = DIMB;
    using Params = KernelParamsBase<Real>;
    using Acc = typename AccFor<Real>::template type<DIMB>;
    using Abs = AccAbs<Real, DIMB>;
    static constexpr int NW = DIMB, NB = DIMB, DOT = 0;   // bounds: the columns
    static LDDMM_D float lgk(const Params& P, float d2) { return lg_factor<KIND, DEG>(P.pk, d2); }
    struct Tgt {
        Real x[D];
    };
    struct Src {
        Real y[D];
        Real b[DIMB];
    };
    static LDDMM_D Real coord(const Tgt& t, int, int j) { return j < D ? t.x[j < D ? j : 0] : (Real)0; }
    static LDDMM_D void lower(const Tgt&, int, const Real* a, Real, Real* lo) {
#pragma unroll
        for (int c = 0; c < DIMB; ++c) lo[c] = a[c];
    }
    static LDDMM_D void upper(const float* lgw, float, float lk, const float*, float* u) {
#pragma unroll
        for (int c = 0; c < DIMB; ++c) u[c] = lgw[c] + lk;
    }
    static LDDMM_D void load_target(const Params& P, long long row, Tgt& t) {
        load_vals<Real, D>(P.tgt4, P.tgt_stride, row, 0, t.x);
    }
    static LDDMM_D void load_source(const float4* S, int j, Src& s) {
        load_vals_smem<Real, D>(S, j, 0, s.y);
        load_vals_smem<Real, DIMB>(S, j, PP, s.b);
    }
    template <bool LIB = false, class A>
    static LDDMM_D void pair(const Params& P, const Tgt& t, const Src& s, A& a) {
        Real r2 = 0;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            const Real dj = t.x[j] - s.y[j];
            r2 = j == 0 ? dj * dj : r2 + dj * dj;
        }
        const Real k = kval<Real, KIND, DEG, LIB>(P.pk, r2);
#pragma unroll
        for (int c = 0; c < DIMB; ++c) a.fma(c, k, s.b[c]);
    }
};

// ---------------------------------------------------------------------------
// f_k = sum_l K'(x_k,y_l) 2 (x_k - y_l) <u_k, v_l>     (up to the epilogue's scale)
// ---------------------------------------------------------------------------
template <class Real_, int KIND, int DEG, int D, int W>
struct OpDiffKT {
    using Real = Real_;
    static constexpr bool F32 = sizeof(Real) == 4;
    static constexpr int FAMILY = KIND;
    static constexpr int TPS = 1;
    static constexpr int R = 2;
    static constexpr int PP = PointPlanes<Real>::N;
    static constexpr int WP = (W + Traits<Real>::PER_WORD - 1) / Traits<Real>::PER_WORD;
    static constexpr int NS = PP + WP;
    static constexpr int NOUT = D;
    using Params = KernelParamsBase<Real>;
    using Acc = typename AccFor<Real>::template type<D>;
    using Abs = AccAbs<Real, D>;
    static constexpr int NW = W, NB = D, DOT = W;   // bounds: the components
    static LDDMM_D float lgk(const Params& P, float d2) { return lg_factor<KIND, DEG>(P.pq, d2); }
    struct Tgt {
        Real x[D];
        Real u[W];
    };
    struct Src {
        Real y[D];
        Real v[W];
    };
    static LDDMM_D Real coord(const Tgt& t, int, int j) { return j < D ? t.x[j < D ? j : 0] : (Real)0; }
    static LDDMM_D Real dot_val(const Tgt& t, int, int w) { return t.u[w]; }
    static LDDMM_D void lower(const Tgt&, int, const Real* a, Real norm1, Real* lo) {
#pragma unroll
        for (int j = 0; j < D; ++j) lo[j] = norm1 == (Real)0 ? (Real)-1 : a[j] / norm1;
    }
    static LDDMM_D void upper(const float*, float lgv, float lk, const float* lext, float* u) {
#pragma unroll
        for (int j = 0; j < D; ++j) u[j] = lgv + lk + lext[j];
    }
    static LDDMM_D void load_target(const Params& P, long long row, Tgt& t) {
        load_vals<Real, D>(P.tgt4, P.tgt_stride, row, 0, t.x);
        load_vals<Real, W>(P.tgt4, P.tgt_stride, row, PP, t.u);
    }
    static LDDMM_D void load_source(const float4* S, int j, Src& s) {
        load_vals_smem<Real, D>(S, j, 0, s.y);
        load_vals_smem<Real, W>(S, j, PP, s.v);
    }
    template <bool LIB = false, class A>
    static LDDMM_D void pair(const Params& P, const Tgt& t, const Src& s, A& a) {
        Real dx[D];
        Real r2 = 0;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            dx[j] = t.x[j] - s.y[j];
            r2 = j == 0 ? dx[j] * dx[j] : r2 + dx[j] * dx[j];
        }
        Real dot = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) dot = w == 0 ? t.u[0] * s.v[0] : dot + t.u[w] * s.v[w];
        const Real g = kdiff<Real, KIND, DEG, LIB>(P.pq, r2) * dot;
#pragma unroll
        for (int j = 0; j < D; ++j) a.fma(j, g, dx[j]);
    }
};

// ---------------------------------------------------------------------------
// div_k = sum_l K'(x_k,y_l) 2 <x_k - y_l, a_l>      (up to the epilogue's scale)
// py-lddmm/kernelFunctions.py:510-530 (applyDivergence)
// ---------------------------------------------------------------------------
template <class Real_, int KIND, int DEG, int D>
struct OpDivergence {
    using Real = Real_;
    static constexpr bool F32 = sizeof(Real) == 4;
    static constexpr int FAMILY = KIND;
    static constexpr int TPS = 1;
    static constexpr int R = 4;
    static constexpr int PP = PointPlanes<Real>::N;
    static constexpr int WP = (D + Traits<Real>::PER_WORD - 1) / Traits<Real>::PER_WORD;
    static constexpr int NS = PP + WP;
    static constexpr int NOUT = 1;
    using Params = KernelParamsBase<Real>;
    using Acc = typename AccFor<Real>::template type<1>;
    struct Tgt {
        Real x[D];
    };
    struct Src {
        Real y[D];
        Real a[D];
    };
    static LDDMM_D void load_target(const Params& P, long long row, Tgt& t) {
        load_vals<Real, D>(P.tgt4, P.tgt_stride, row, 0, t.x);
    }
    static LDDMM_D void load_source(const float4* S, int j, Src& s) {
        load_vals_smem<Real, D>(S, j, 0, s.y);
        load_vals_smem<Real, D>(S, j, PP, s.a);
    }
    template <bool LIB = false>
    static LDDMM_D void pair(const Params& P, const Tgt& t, const Src& s, Acc& acc) {
        Real r2 = 0, dot = 0;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            const Real dj = t.x[j] - s.y[j];
            r2 = j == 0 ? dj * dj : r2 + dj * dj;
            dot = j == 0 ? dj * s.a[j] : dot + dj * s.a[j];
        }
        acc.fma(0, kdiff<Real, KIND, DEG, LIB>(P.pq, r2), dot);
    }
};

}  // namespace lddmm
