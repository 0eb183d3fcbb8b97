// Data-term operators and helper kernels shared by dataterms.cu (single
// problem) and ragged.cu (many requests per launch).  Formulas and reference
// lines: see dataterms.cu.
#pragma once
#include <type_traits>

#include "host.h"
#include "ops2.cuh"
#include "pack.cuh"
#include "sweep_dispatch.cuh"

namespace lddmm {

enum DataNorm : int { NCURRENT = 0, NMEASURE = 1, NVARIFOLD = 2 };
enum DataMode : int { M_VARI_VALUE = 0, M_VARI_GRAD = 1, M_CUR_GRAD = 2, M_MEAS_GRAD = 3 };

// Gaussian K' uses the same exponential as K.
template <class Real, int KIND, int PDEG, int QDEG, bool LIB>
LDDMM_D void kboth(const Real* pk, const Real* pq, Real r2, Real& k, Real& f) {
    if constexpr (KIND == KGAUSS) {
        k = kval<Real, KIND, 0, LIB>(pk, r2);
        f = k;
    } else if constexpr (sizeof(Real) == 4) {
        const float u = sqrt_approx(r2);
        const float e = ex2(-u);
        k = (PDEG == 0 ? 1.f : horner<PDEG>(pk, u)) * e;
        f = (QDEG == 0 ? pq[0] : horner<QDEG>(pq, u)) * e;
    } else {
        const double u = sqrt(r2);
        const bool zero = LIB ? u < kZeroThresh : less_nonneg(u, kZero2Lap);
        const double e = LIB ? exp(-1.0 * u) : exp2neg(u);
        k = zero ? 1.0 : poly64<PDEG>(pk, u) * e;
        f = zero ? pq[0] : poly64<QDEG>(pq, u) * e;
    }
}

template <int MODE, int D>
struct DataLayout {
    static constexpr int TV = (MODE == M_VARI_VALUE || MODE == M_VARI_GRAD) ? 3 : (MODE == M_CUR_GRAD ? D : 0);
    static constexpr int SV = (MODE == M_VARI_VALUE || MODE == M_VARI_GRAD) ? 4 : (MODE == M_CUR_GRAD ? D : 1);
    static constexpr int NOUT = MODE == M_VARI_VALUE ? 1
                                : MODE == M_VARI_GRAD ? 2 * D + 1
                                : MODE == M_CUR_GRAD  ? 2 * D
                                                      : D + 1;
};

// Bounds of the data-term sweeps (see op_culls, sweep.cuh).  Weight columns: the weight
// (varifold value, measure), the components of the vector (current), or those of the
// weighted normal and the weight (varifold gradient).
constexpr int dt_weights(int mode, int D) { return mode == M_VARI_GRAD ? D + 1 : mode == M_CUR_GRAD ? D : 1; }

// What the sums of a target with values u hold at least.  Varifold gradient: its sums
// 0..D-1 and D meet in z1_j = a_j + a_D u_j, so what is left out of either has to be small
// against |a_j| + |a_D u_j| (near flat pieces a_D is next to nothing by itself).
template <int MODE, int D, class Real>
LDDMM_D void dt_lower(const Real* u, const Real* a, Real norm1, Real* lo) {
    if constexpr (MODE == M_VARI_GRAD) {
        lo[D] = -1;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            const Real n = u[j] < (Real)0 ? -u[j] : u[j];
            lo[j] = a[j] + a[D] * n;
            if (n != (Real)0) {
                const Real q = lo[j] / n;
                if (!(lo[D] >= (Real)0) || !(q >= lo[D])) lo[D] = lo[D] != lo[D] ? lo[D] : q;
            }
            lo[D + 1 + j] = a[D + 1 + j];
        }
    } else {
#pragma unroll
        for (int b = 0; b < DataLayout<MODE, D>::NOUT; ++b) lo[b] = a[b];
        if constexpr (MODE == M_CUR_GRAD)
#pragma unroll
            for (int j = 0; j < D; ++j) lo[D + j] = norm1 == (Real)0 ? (Real)-1 : a[D + j] / norm1;
    }
}
template <int MODE, int D>
LDDMM_D void dt_upper(const float* lgw, float lgv, float lk, const float* lext, float* u) {
    if constexpr (MODE == M_VARI_VALUE) {
        u[0] = lgw[0] + lk + 1.f;                       // 1 + <n, n'>^2 <= 2
    } else if constexpr (MODE == M_VARI_GRAD) {
#pragma unroll
        for (int j = 0; j < D; ++j) {
            u[j] = lgw[j] + lk + 2.f;                   // 2 <n, n'>, and half of what z1_j may lose
            u[D + 1 + j] = lgw[D] + lk + 1.f + lext[j];
        }
        u[D] = lgw[D] + lk + 1.f;                       // the other half
    } else if constexpr (MODE == M_CUR_GRAD) {
#pragma unroll
        for (int j = 0; j < D; ++j) {
            u[j] = lgw[j] + lk;
            u[D + j] = lgv + lk + lext[j];
        }
    } else {
        u[0] = lgw[0] + lk;
#pragma unroll
        for (int j = 0; j < D; ++j) u[1 + j] = lgw[0] + lk + lext[j];
    }
}
// the half h of N packed values
template <int N>
LDDMM_D void halves2(const f2* v, int h, float* out) {
#pragma unroll
    for (int j = 0; j < N; ++j) out[j] = half2(v[j], h);
}

template <class Real_, int KIND, int PDEG, int QDEG, int D, int MODE>
struct OpData {
    using Real = Real_;
    using L = DataLayout<MODE, D>;
    static constexpr bool F32 = sizeof(Real) == 4;
    static constexpr int FAMILY = KIND;
    static constexpr int TPS = 1;
    static constexpr int R = 2;
    static constexpr int PP = PointPlanes<Real>::N;
    static constexpr int PW = Traits<Real>::PER_WORD;
    static constexpr int TVW = (L::TV + PW - 1) / PW;
    static constexpr int SVW = (L::SV + PW - 1) / PW;
    static constexpr int NT = PP + TVW;  // target planes
    static constexpr int NS = PP + SVW;  // source planes
    static constexpr int NOUT = L::NOUT;
    using Params = KernelParamsBase<Real>;
    using Acc = typename AccFor<Real>::template type<NOUT>;
    using Abs = AccAbs<Real, NOUT>;
    static constexpr int NW = dt_weights(MODE, D), NB = NOUT, DOT = MODE == M_CUR_GRAD ? D : 0;
    // K bounds the factor of K' as well (its polynomial Q is below P term by term)
    static LDDMM_D float lgk(const Params& P, float d2) { return lg_factor<KIND, PDEG>(P.pk, d2); }
    struct Tgt {
        Real x[D];
        Real u[L::TV > 0 ? L::TV : 1];
    };
    struct Src {
        Real y[D];
        Real v[L::SV];
    };
    static LDDMM_D Real coord(const Tgt& t, int, int j) { return j < D ? t.x[j < D ? j : 0] : (Real)0; }
    static LDDMM_D Real dot_val(const Tgt& t, int, int w) { return t.u[w]; }
    static LDDMM_D void lower(const Tgt& t, int, const Real* a, Real norm1, Real* lo) { dt_lower<MODE, D>(t.u, a, norm1, lo); }
    static LDDMM_D void upper(const float* lgw, float lgv, float lk, const float* lext, float* u) {
        dt_upper<MODE, D>(lgw, lgv, lk, lext, u);
    }
    static LDDMM_D void load_target(const Params& P, long long row, Tgt& t) {
        load_vals<Real, D>(P.tgt4, P.tgt_stride, row, 0, t.x);
        if constexpr (L::TV > 0) load_vals<Real, L::TV>(P.tgt4, P.tgt_stride, row, PP, t.u);
    }
    static LDDMM_D void load_source(const float4* S, int j, Src& s) {
        load_vals_smem<Real, D>(S, j, 0, s.y);
        load_vals_smem<Real, L::SV>(S, j, PP, s.v);
    }
    template <bool LIB = false, class A>
    static LDDMM_D void pair(const Params& P, const Tgt& t, const Src& s, A& acc) {
        Real dx[D], r2 = 0;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            dx[j] = t.x[j] - s.y[j];
            r2 = j == 0 ? dx[j] * dx[j] : r2 + dx[j] * dx[j];
        }
        if constexpr (MODE == M_VARI_VALUE) {
            const Real k = kval<Real, KIND, PDEG, LIB>(P.pk, r2);
            const Real dn = t.u[0] * s.v[0] + t.u[1] * s.v[1] + t.u[2] * s.v[2];
            acc.fma(0, k * s.v[3], (Real)1 + dn * dn);
        } else {
            Real k, f;
            kboth<Real, KIND, PDEG, QDEG, LIB>(P.pk, P.pq, r2, k, f);
            if constexpr (MODE == M_VARI_GRAD) {
                const Real dn = t.u[0] * s.v[0] + t.u[1] * s.v[1] + t.u[2] * s.v[2];
                const Real wk = k * s.v[3];
                const Real ca = 2 * dn * wk;
#pragma unroll
                for (int j = 0; j < D; ++j) acc.fma(j, ca, s.v[j]);
                acc.fma(D, wk, (Real)1 - dn * dn);
                const Real wf = f * s.v[3] * ((Real)1 + dn * dn);
#pragma unroll
                for (int j = 0; j < D; ++j) acc.fma(D + 1 + j, wf, dx[j]);
            } else if constexpr (MODE == M_CUR_GRAD) {
                Real dot = 0;
#pragma unroll
                for (int j = 0; j < D; ++j) {
                    acc.fma(j, k, s.v[j]);
                    dot = j == 0 ? t.u[0] * s.v[0] : dot + t.u[j] * s.v[j];
                }
                const Real g = f * dot;
#pragma unroll
                for (int j = 0; j < D; ++j) acc.fma(D + j, g, dx[j]);
            } else {  // M_MEAS_GRAD
                acc.fma(0, k, s.v[0]);
                const Real g = f * s.v[0];
#pragma unroll
                for (int j = 0; j < D; ++j) acc.fma(1 + j, g, dx[j]);
            }
        }
    }
};

// Packed-pair FP32 varifold VALUE operator (two targets per thread slot, see
// ops2.cuh): the per-pair arithmetic of OpData<float, ..., M_VARI_VALUE>
//   acc += K(c_k, c_l) (1 + <n_k, n_l>^2) w_l
// with sources stored as list records [y0 y1 y2 n0 n1 n2 w] (2 words)
// and targets in the standard planes (pos word, normal word).  d = 3 only.
template <int KIND, int PDEG>
struct OpVariValue2 {
    using Real = float;
    static constexpr bool F32 = true;
    static constexpr bool LIST = true;
    static constexpr int TPS = 2;
    static constexpr int R = 4;
    static constexpr int PP = 1;
    static constexpr int NV = 7;
    static constexpr int NS = (NV + 3) / 4;
    static constexpr int NOUT = 1;
    using Params = KernelParams2;
    using Acc = AccF32C2<1>;
    using Abs = AccAbs2<NOUT>;
    static constexpr int NW = dt_weights(M_VARI_VALUE, 3), NB = NOUT, DOT = 0;
    static LDDMM_D float lgk(const Params& P, float d2) { return lg_factor<KIND, PDEG>(P.pkd, d2); }
    struct Tgt {
        f2 x[3];
        f2 u[3];
    };
    struct Src {
        f2 val[NV];
    };
    static LDDMM_D float coord(const Tgt& t, int h, int j) { return half2(t.x[j], h); }
    static LDDMM_D float dot_val(const Tgt& t, int h, int w) { return half2(t.u[w], h); }
    static LDDMM_D void lower(const Tgt& t, int h, const float* a, float norm1, float* lo) {
        float u[3];
        halves2<3>(t.u, h, u);
        dt_lower<M_VARI_VALUE, 3>(u, a, norm1, lo);
    }
    static LDDMM_D void upper(const float* lgw, float lgv, float lk, const float* lext, float* u) {
        dt_upper<M_VARI_VALUE, 3>(lgw, lgv, lk, lext, u);
    }
    static LDDMM_D void load_target(const Params& P, long long ra, long long rb, Tgt& t) {
        load_target_pair<3>(P.tgt4, P.tgt_stride, ra, rb, 0, t.x);
        load_target_pair<3>(P.tgt4, P.tgt_stride, ra, rb, 1, t.u);
    }
    static LDDMM_D void load_source(const float4* S, int j, Src& s) { load_list_source<NV>(S, j, s.val); }
    template <class A>
    static LDDMM_D void pair(const Params& P, const Tgt& t, const Src& s, A& a) {
        f2 r2;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const f2 dj = sub2(t.x[j], s.val[j]);
            r2 = j == 0 ? mul2(dj, dj) : fma2(dj, dj, r2);
        }
        const f2 k = kval2<KIND, PDEG>(P.pkd, r2);
        const f2 dn = fma2(t.u[2], s.val[5], fma2(t.u[1], s.val[4], mul2(t.u[0], s.val[3])));
        const f2 q = fma2(dn, dn, splat2(1.f));
        a.fma(0, mul2(k, s.val[6]), q);
    }
};

// Packed-pair FP32 varifold GRADIENT operator: the arithmetic of
// OpData<float, ..., M_VARI_GRAD> for two target cells per slot (sources as in
// OpVariValue2, weights carrying the -1 of the target shape):
//   acc[0..3) += 2 <n_k,n_l> K w_l n_l,  acc[3] += K w_l (1 - <n_k,n_l>^2),
//   acc[4..7) += K' w_l (1 + <n_k,n_l>^2) (c_k - c_l)'
// 21 packed instructions per slot and source (Gaussian): acc[0..3) is summed
// without its factor 2 (restored exactly by out_scale when written), and
// 1 - <n,n'>^2 is formed as 2 - (1 + <n,n'>^2) from the factor the K' part needs.
// Two packed slots per thread (R = 4): each 2-word source record read from
// shared memory serves four target cells.
template <int KIND, int PDEG, int QDEG>
struct OpVariGrad2 {
    using Real = float;
    static constexpr bool F32 = true;
    static constexpr bool LIST = true;
    static constexpr int TPS = 2;
    static constexpr int R = 4;
    static constexpr int PP = 1;
    static constexpr int NV = 7;
    static constexpr int NS = (NV + 3) / 4;
    static constexpr int NOUT = 7;
    using Params = KernelParams2;
    using Acc = AccF32C2<NOUT>;
    using Abs = AccAbs2<NOUT>;
    static constexpr int NW = dt_weights(M_VARI_GRAD, 3), NB = NOUT, DOT = 0;
    static LDDMM_D float lgk(const Params& P, float d2) { return lg_factor<KIND, PDEG>(P.pkd, d2); }
    struct Tgt {
        f2 x[3];
        f2 u[3];
    };
    struct Src {
        f2 val[NV];
    };
    static LDDMM_D float coord(const Tgt& t, int h, int j) { return half2(t.x[j], h); }
    static LDDMM_D float dot_val(const Tgt& t, int h, int w) { return half2(t.u[w], h); }
    static LDDMM_D void lower(const Tgt& t, int h, const float* a, float norm1, float* lo) {
        float u[3];
        halves2<3>(t.u, h, u);
        dt_lower<M_VARI_GRAD, 3>(u, a, norm1, lo);
    }
    static LDDMM_D void upper(const float* lgw, float lgv, float lk, const float* lext, float* u) {
        dt_upper<M_VARI_GRAD, 3>(lgw, lgv, lk, lext, u);
    }
    static LDDMM_D void load_target(const Params& P, long long ra, long long rb, Tgt& t) {
        load_target_pair<3>(P.tgt4, P.tgt_stride, ra, rb, 0, t.x);
        load_target_pair<3>(P.tgt4, P.tgt_stride, ra, rb, 1, t.u);
    }
    static LDDMM_D void load_source(const float4* S, int j, Src& s) { load_list_source<NV>(S, j, s.val); }
    template <class A>
    static LDDMM_D void pair(const Params& P, const Tgt& t, const Src& s, A& a) {
        f2 dx[3], r2;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            dx[j] = sub2(t.x[j], s.val[j]);
            r2 = j == 0 ? mul2(dx[j], dx[j]) : fma2(dx[j], dx[j], r2);
        }
        f2 k, f;
        if constexpr (KIND == KGAUSS) {
            k = kval2<KIND, PDEG>(P.pkd, r2);
            f = k;
        } else {
            const f2 u = sqrt2(r2);
            const f2 e = ex2neg2(u);
            k = PDEG == 0 ? e : mul2(horner2<PDEG>(P.pkd, u), e);
            f = QDEG == 0 ? mul2(f2{P.pqd[0]}, e) : mul2(horner2<QDEG>(P.pqd, u), e);
        }
        const f2 dn = fma2(t.u[2], s.val[5], fma2(t.u[1], s.val[4], mul2(t.u[0], s.val[3])));
        const f2 wk = mul2(k, s.val[6]);
        const f2 ca = mul2(dn, wk);                       // half of 2 <n,n'> K w
#pragma unroll
        for (int j = 0; j < 3; ++j) a.fma(j, ca, s.val[3 + j]);
        const f2 q1 = fma2(dn, dn, splat2(1.f));          // 1 + <n,n'>^2
        a.fma(3, wk, sub2(splat2(2.f), q1));              // 1 - <n,n'>^2
        const f2 wf = mul2(KIND == KGAUSS ? wk : mul2(f, s.val[6]), q1);
#pragma unroll
        for (int j = 0; j < 3; ++j) a.fma(4 + j, wf, dx[j]);
    }
    static LDDMM_D double out_scale(int c) { return c < 3 ? 2.0 : 1.0; }
};

// Packed-pair FP32 current GRADIENT operator (OpData<float, ..., M_CUR_GRAD>,
// d = 3): sources [y0 y1 y2 s0 s1 s2], targets (pos, s_k):
//   acc[0..3) += K s_l,  acc[3..6) += K' <s_k, s_l> (c_k - c_l)'
template <int KIND, int PDEG, int QDEG>
struct OpCurGrad2 {
    using Real = float;
    static constexpr bool F32 = true;
    static constexpr bool LIST = true;
    static constexpr int TPS = 2;
    static constexpr int R = 2;
    static constexpr int PP = 1;
    static constexpr int NV = 6;
    static constexpr int NS = (NV + 3) / 4;
    static constexpr int NOUT = 6;
    using Params = KernelParams2;
    using Acc = AccF32C2<NOUT>;
    using Abs = AccAbs2<NOUT>;
    static constexpr int NW = dt_weights(M_CUR_GRAD, 3), NB = NOUT, DOT = 3;
    static LDDMM_D float lgk(const Params& P, float d2) { return lg_factor<KIND, PDEG>(P.pkd, d2); }
    struct Tgt {
        f2 x[3];
        f2 u[3];
    };
    struct Src {
        f2 val[NV];
    };
    static LDDMM_D float coord(const Tgt& t, int h, int j) { return half2(t.x[j], h); }
    static LDDMM_D float dot_val(const Tgt& t, int h, int w) { return half2(t.u[w], h); }
    static LDDMM_D void lower(const Tgt& t, int h, const float* a, float norm1, float* lo) {
        float u[3];
        halves2<3>(t.u, h, u);
        dt_lower<M_CUR_GRAD, 3>(u, a, norm1, lo);
    }
    static LDDMM_D void upper(const float* lgw, float lgv, float lk, const float* lext, float* u) {
        dt_upper<M_CUR_GRAD, 3>(lgw, lgv, lk, lext, u);
    }
    static LDDMM_D void load_target(const Params& P, long long ra, long long rb, Tgt& t) {
        load_target_pair<3>(P.tgt4, P.tgt_stride, ra, rb, 0, t.x);
        load_target_pair<3>(P.tgt4, P.tgt_stride, ra, rb, 1, t.u);
    }
    static LDDMM_D void load_source(const float4* S, int j, Src& s) { load_list_source<NV>(S, j, s.val); }
    template <class A>
    static LDDMM_D void pair(const Params& P, const Tgt& t, const Src& s, A& a) {
        f2 dx[3], r2;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            dx[j] = sub2(t.x[j], s.val[j]);
            r2 = j == 0 ? mul2(dx[j], dx[j]) : fma2(dx[j], dx[j], r2);
        }
        f2 k, f;
        if constexpr (KIND == KGAUSS) {
            k = kval2<KIND, PDEG>(P.pkd, r2);
            f = k;
        } else {
            const f2 u = sqrt2(r2);
            const f2 e = ex2neg2(u);
            k = PDEG == 0 ? e : mul2(horner2<PDEG>(P.pkd, u), e);
            f = QDEG == 0 ? mul2(f2{P.pqd[0]}, e) : mul2(horner2<QDEG>(P.pqd, u), e);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) a.fma(j, k, s.val[3 + j]);
        const f2 dot = fma2(t.u[2], s.val[5], fma2(t.u[1], s.val[4], mul2(t.u[0], s.val[3])));
        const f2 g = mul2(f, dot);
#pragma unroll
        for (int j = 0; j < 3; ++j) a.fma(3 + j, g, dx[j]);
    }
};

// Packed operators (LIST) take duplicated polynomial coefficients and list
// source records from the pack.
template <class Op, class = void>
struct op_list : std::false_type {};
template <class Op>
struct op_list<Op, std::void_t<decltype(Op::LIST)>> : std::bool_constant<Op::LIST> {};

// ---- geometry -----------------------------------------------------------------
// centres (nc, d), vectors (nc, d) (surfels or tangents) of set 1; invalid cell
// indices give zero geometry (host code validates them before the call).
static __global__ void cell_geometry_kernel(int ncorner, const double* __restrict__ v, long long nv, int d,
                                            const int64_t* __restrict__ cells, long long nc, double* __restrict__ c,
                                            double* __restrict__ s) {
    for (long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x; f < nc;
         f += (long long)gridDim.x * blockDim.x) {
        long long id[3] = {0, 0, 0};
        bool ok = true;
        for (int q = 0; q < ncorner; ++q) {
            id[q] = cells[f * ncorner + q];
            ok = ok && id[q] >= 0 && id[q] < nv;
        }
        if (!ok) {
            for (int j = 0; j < d; ++j) c[f * d + j] = s[f * d + j] = 0.0;
            continue;
        }
        const double* x0 = v + id[0] * d;
        const double* x1 = v + id[1] * d;
        if (ncorner == 3) {
            const double* x2 = v + id[2] * d;
            for (int j = 0; j < 3; ++j) c[f * 3 + j] = (x0[j] + x1[j] + x2[j]) / 3;
            const double e1[3] = {x1[0] - x0[0], x1[1] - x0[1], x1[2] - x0[2]};
            const double e2[3] = {x2[0] - x0[0], x2[1] - x0[1], x2[2] - x0[2]};
            s[f * 3 + 0] = e1[1] * e2[2] - e1[2] * e2[1];
            s[f * 3 + 1] = e1[2] * e2[0] - e1[0] * e2[2];
            s[f * 3 + 2] = e1[0] * e2[1] - e1[1] * e2[0];
        } else {
            for (int j = 0; j < d; ++j) {
                c[f * d + j] = (x0[j] + x1[j]) / 2;
                s[f * d + j] = x1[j] - x0[j];
            }
        }
    }
}

LDDMM_D double vec_norm_eps(const double* s, int d, double eps) {
    double q = 0.0;
    for (int j = 0; j < d; ++j) q += s[j] * s[j];
    return sqrt(q + eps);
}

// One packed record of a data-term sweep (row i of `planes`, stride words per
// plane): the prescaled centre, then the values of the norm:
//   norm current : target -, source s*sign              (value, OpApplyK DIMB = d)
//                  target s, source s*sign              (gradient)
//   norm measure : target -, source a*sign              (value and gradient)
//   norm varifold: target n, source (n, a*sign)         (value and gradient)
// c == nullptr writes a zero (padding) record of nplanes planes.
// bp, bw (sources): the packed position and the columns that bound what the record adds (dt_weights of them).
template <class Real>
LDDMM_D void dt_pack_record(int norm, int grad, bool is_t, const double* c, const double* s, int d, double eps,
                            double sign, double scale, const double* center, float4* planes, long long stride,
                            long long i, int nplanes, int slots, bool list = false, Real* bp = nullptr,
                            Real* bw = nullptr) {
    constexpr int PP = PointPlanes<Real>::N;
    if (c == nullptr) {
        if (bp != nullptr) {
            for (int j = 0; j < 3; ++j) bp[j] = 0;
            for (int j = 0; j < 4; ++j) bw[j] = 0;
        }
        for (int p = 0; p < nplanes; ++p) planes[(long long)p * stride + i] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const double a = vec_norm_eps(s, d, eps);
    double pos[4] = {0, 0, 0, 0};
    for (int j = 0; j < d; ++j) pos[j] = (c[j] - center[j]) * scale;
    if (bp != nullptr) {
        for (int j = 0; j < 3; ++j) bp[j] = (Real)pos[j];
        for (int j = 0; j < 4; ++j) bw[j] = 0;
        if (norm == NCURRENT) {
            for (int j = 0; j < d; ++j) bw[j] = (Real)(s[j] * sign);
        } else if (norm == NVARIFOLD && grad) {
            for (int j = 0; j < 3; ++j) bw[j] = (Real)(s[j] / a) * (Real)(a * sign);
            bw[3] = (Real)(a * sign);
        } else {
            bw[0] = (Real)(a * sign);
            // 0 / 0 of a cell without area: never passed over, though it weighs nothing
            if (norm == NVARIFOLD) bw[0] += (Real)(s[0] / a + s[1] / a + s[2] / a) * (Real)0;
        }
    }
    if (sizeof(Real) == 4 && list) {
        // list source record [pos0 pos1 pos2 vals...] (see ops2.cuh)
        double vals[4] = {0, 0, 0, 0};
        if (norm == NVARIFOLD) {
            for (int j = 0; j < 3; ++j) vals[j] = s[j] / a;
            vals[3] = a * sign;
        } else if (norm == NCURRENT) {
            for (int j = 0; j < d; ++j) vals[j] = s[j] * sign;
        } else {
            vals[0] = a * sign;
        }
        float q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int j = 0; j < 3; ++j) q[j] = (float)pos[j];
        for (int j = 0; j < slots && j < 4; ++j) q[3 + j] = (float)vals[j];
        for (int w = 0; w < nplanes; ++w)
            planes[(long long)w * stride + i] = make_float4(q[4 * w], q[4 * w + 1], q[4 * w + 2], q[4 * w + 3]);
        return;
    }
    if constexpr (sizeof(Real) == 4) {
        planes[i] = make_float4((float)pos[0], (float)pos[1], (float)pos[2], 0.f);
    } else {
        double2* o = reinterpret_cast<double2*>(planes);
        o[i] = make_double2(pos[0], pos[1]);
        o[stride + i] = make_double2(pos[2], 0.0);
    }
    double vals[4] = {0, 0, 0, 0};
    int nv = 0;
    if (norm == NVARIFOLD) {
        for (int j = 0; j < 3; ++j) vals[j] = s[j] / a;
        nv = 3;
        if (!is_t) {
            vals[3] = a * sign;
            nv = 4;
        }
    } else if (norm == NCURRENT) {
        if (!is_t || grad) {
            for (int j = 0; j < d; ++j) vals[j] = s[j] * sign;
            nv = d;
        }
    } else {
        if (!is_t) {
            vals[0] = a * sign;
            nv = 1;
        }
    }
    constexpr int PWv = Traits<Real>::PER_WORD;
    for (int w = 0; w < (slots + PWv - 1) / PWv; ++w) {
        Real q[PWv];
        for (int j = 0; j < PWv; ++j) q[j] = (w * PWv + j < nv) ? (Real)vals[w * PWv + j] : (Real)0;
        float4* dst = planes + (long long)(PP + w) * stride + i;
        if constexpr (sizeof(Real) == 4) *dst = make_float4(q[0], q[1], q[2], q[3]);
        else *reinterpret_cast<double2*>(dst) = make_double2(q[0], q[1]);
    }
}

// Targets: set-1 cells.  Sources: set-1 cells (sign +1) then set-2 cells (sign2).
template <class Real>
static __global__ void dt_pack_kernel(int norm, int grad, const double* __restrict__ c1, const double* __restrict__ s1,
                                      long long n1, const double* __restrict__ c2, const double* __restrict__ s2,
                                      long long n2, int d, double eps1, double eps2, double sign2, double scale,
                                      const double* __restrict__ center, float4* tgt, long long tstride, int tplanes,
                                      int tslots, float4* src, long long sstride, int splanes, int sslots,
                                      int list, long long n1s, float4* boxes, int nw, int* __restrict__ counters,
                                      int n_counters) {
    // set-2 sources start at row n1s (n1 rounded up to a fold for symmetric sweeps)
    const long long npad = tstride > sstride ? tstride : sstride;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npad;
         i += (long long)gridDim.x * blockDim.x) {
        if (i < n_counters) counters[i] = 0;
        if (i < tstride)
            dt_pack_record<Real>(norm, grad, true, i < n1 ? c1 + i * d : nullptr, i < n1 ? s1 + i * d : nullptr, d,
                                 eps1, 1.0, scale, center, tgt, tstride, i, tplanes, tslots);
        if (i < sstride) {
            const bool first = i < n1, second = i >= n1s && i < n1s + n2;
            const double* c = first ? c1 + i * d : (second ? c2 + (i - n1s) * d : nullptr);
            const double* sv = first ? s1 + i * d : (second ? s2 + (i - n1s) * d : nullptr);
            Real bp[3], bw[4];
            dt_pack_record<Real>(norm, grad, false, c, sv, d, first ? eps1 : eps2, first ? 1.0 : sign2, scale, center,
                                 src, sstride, i, splanes, sslots, list != 0, bp, bw);
            if (boxes != nullptr) store_fold_box<Real, 4>(boxes, i, c != nullptr, bp, bw, nw);
        }
    }
}

// per-cell z1, dz1 of row i from the chunk sums of its sums
LDDMM_D void dt_grad_row(int norm, const double* acc, const double* s, int d, double eps1, double dzscale, double* z1,
                         double* dz1) {
    if (norm == NCURRENT) {
        for (int j = 0; j < d; ++j) {
            z1[j] = acc[j];
            dz1[j] = dzscale * acc[d + j];
        }
    } else if (norm == NMEASURE) {
        const double a = vec_norm_eps(s, d, eps1);
        for (int j = 0; j < d; ++j) {
            z1[j] = acc[0] * (s[j] / a);
            dz1[j] = dzscale * a * acc[1 + j];
        }
    } else {
        const double a = vec_norm_eps(s, d, eps1);
        for (int j = 0; j < d; ++j) {
            z1[j] = acc[j] + acc[d] * (s[j] / a);
            dz1[j] = dzscale * a * acc[d + 1 + j];
        }
    }
}

// what a cell adds to the energy: w1 . z (current: s1 . z, measure and varifold: a1 z)
LDDMM_D double dt_value_row(int norm, const double* z, const double* s, int d, double eps1) {
    if (norm != NCURRENT) return vec_norm_eps(s, d, eps1) * z[0];
    double e = 0.0;
    for (int j = 0; j < d; ++j) e += s[j] * z[j];
    return e;
}

// Epilogue of the value sweeps: energy partial of the group's cells; the last group adds them.
struct EpiDtValue {
    static constexpr bool NONE = false;
    int norm;
    const double* s1;
    int d;
    double eps1;
    double* epart;
    int groups;
    int* counter;
    double* energy;
    template <int GT, int NOUT>
    LDDMM_D void run(const SegDesc& sg, int tb, const int* srow, const double* red) const {
        double e = 0.0;
        for (int r = threadIdx.x; r < GT; r += blockDim.x) {
            const long long i = srow[r];
            if (i < sg.n_tgt) e += dt_value_row(norm, red + r * NOUT, s1 + i * d, d, eps1);
        }
        e = block_sum_all(e);
        if (threadIdx.x == 0) epart[tb] = e;
        if (!last_block(counter, groups)) return;
        e = 0.0;
        for (int q = threadIdx.x; q < groups; q += blockDim.x) e += __ldcg(epart + q);
        e = block_sum_all(e);
        if (threadIdx.x == 0) *energy = e;
    }
};

// Epilogue of the gradient sweeps: per-cell z1, dz1.
struct EpiDtGrad {
    static constexpr bool NONE = false;
    int norm;
    const double* s1;
    int d;
    double eps1, dzscale;
    double *z1, *dz1;
    template <int GT, int NOUT>
    LDDMM_D void run(const SegDesc& sg, int, const int* srow, const double* red) const {
        for (int r = threadIdx.x; r < GT; r += blockDim.x) {
            const long long i = srow[r], q = i * d;
            if (i >= sg.n_tgt) continue;
            dt_grad_row(norm, red + r * NOUT, s1 + q, d, eps1, dzscale, z1 + q, dz1 + q);
        }
    }
};

// px[q] = 2 sum over the (cell, corner) entries of vertex q of the corner contribution.
// L2ONLY: z1 / dz1 were written by other CTAs of the same launch (loads bypass L1).
template <bool L2ONLY = false>
LDDMM_D void dt_gather_vertex(long long q, int ncorner, const double* __restrict__ v, long long nv, int d,
                              const int64_t* __restrict__ cells, long long nc, const int64_t* __restrict__ vptr,
                              const int64_t* __restrict__ vidx, const double* z1, const double* dz1,
                              double* __restrict__ px) {
    double acc[3] = {0, 0, 0};
    const long long b = vptr[q], e = vptr[q + 1];
    for (long long k = b; k < e; ++k) {
        const long long code = vidx[k];
        if (code < 0 || code >= nc * ncorner) continue;
        const long long f = code / ncorner;
        const int corner = (int)(code - f * ncorner);
        double z[3] = {0, 0, 0}, dz[3] = {0, 0, 0};
        for (int j = 0; j < d; ++j) {
            z[j] = L2ONLY ? __ldcg(z1 + f * d + j) : z1[f * d + j];
            dz[j] = L2ONLY ? __ldcg(dz1 + f * d + j) : dz1[f * d + j];
        }
        if (ncorner == 3) {
            // opposite edge of the corner: x2-x1, x0-x2, x1-x0
            const int ia = (corner + 2) % 3, ib = (corner + 1) % 3;
            const long long va = cells[f * 3 + ia], vb = cells[f * 3 + ib];
            if (va < 0 || va >= nv || vb < 0 || vb >= nv) continue;
            double ed[3];
            for (int j = 0; j < 3; ++j) ed[j] = v[va * 3 + j] - v[vb * 3 + j];
            const double cr[3] = {ed[1] * z[2] - ed[2] * z[1], ed[2] * z[0] - ed[0] * z[2],
                                  ed[0] * z[1] - ed[1] * z[0]};
            for (int j = 0; j < 3; ++j) acc[j] += dz[j] - cr[j];
        } else {
            const double sgn = corner == 0 ? -1.0 : 1.0;
            for (int j = 0; j < d; ++j) acc[j] += dz[j] + sgn * z[j];
        }
    }
    for (int j = 0; j < d; ++j) px[q * d + j] = 2 * acc[j];
}

static __global__ void dt_gather_kernel(int ncorner, const double* __restrict__ v, long long nv, int d,
                                        const int64_t* __restrict__ cells, long long nc,
                                        const int64_t* __restrict__ vptr, const int64_t* __restrict__ vidx,
                                        const double* __restrict__ z1, const double* __restrict__ dz1,
                                        double* __restrict__ px) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < nv;
         q += (long long)gridDim.x * blockDim.x)
        dt_gather_vertex(q, ncorner, v, nv, d, cells, nc, vptr, vidx, z1, dz1, px);
}


}  // namespace lddmm
