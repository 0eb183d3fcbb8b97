// Packed-pair (two targets per thread slot) FP32 operators for sweep_kernel.
//
//   OpApplyK2<KIND, DEG, D, DIMB>  f_k = sum_l K(x_k,y_l) beta_l        (kernelFunctions.f90:1-54)
//   OpDiffKT2<KIND, DEG, D, W>     f_k = sum_l K'(x_k,y_l) 2(x_k-y_l) <u_k,v_l>  (kernelFunctions.f90:56-114)
//
// Same arithmetic as OpApplyK / OpDiffKT<float> (ops.cuh), evaluated for two
// targets at once with `f32x2` instructions.  Layouts:
//   targets : the standard planes (pos word, then values 4 per word);
//   sources : "list" records, the value list [y_0..y_{D-1}, v_0..v_{V-1}], four
//             values per 16-byte word; splat2 makes the packed operand (v, v) of
//             the f32x2 instructions from each.
//
// Records that hold each value twice, (v, v), need no splat but three words
// instead of two for a Gaussian applyK (four instead of two for the varifold
// operators): more shared-memory reads and more registers in flight per source.
// Measured at n = m = 131,072 (pairs/s, doubled -> single values, 8 sources
// unrolled): Gaussian applyK 2.78 -> 3.02e12, Laplacian 1.84 -> 1.93e12, Gaussian
// applyDiffKT 2.02 -> 2.15e12, adjoint (W = 6) 1.62 -> 1.73e12, varifold value
// 2.36 -> 2.47e12, varifold gradient 1.25 -> 1.33e12, current gradient 1.51 ->
// 1.63e12.  Eight targets per thread instead of four gain nothing more and make
// the groups coarser.  What bounds the sweeps now is the FMA pipe, 80% (Gaussian)
// and 74-76% (Laplacian, with the XU 74-87%) busy, math-pipe throttle the first
// stall.
#pragma once
#include <cstring>

#include "f32x2.cuh"
#include "ops.cuh"
#include "pack.cuh"

namespace lddmm {

struct KernelParams2 {
    const float4* src4;
    long long src_stride;
    const float4* tgt4;
    long long tgt_stride;
    unsigned long long pkd[5];  // K polynomial, each coefficient duplicated as an f32x2 pair
    unsigned long long pqd[4];  // K' polynomial, duplicated
};

// List record j of a fold: NV values, each splat over the two lanes.
template <int NV>
LDDMM_D void load_list_source(const float4* S, int j, f2* val) {
#pragma unroll
    for (int w = 0; w < (NV + 3) / 4; ++w) {
        const float4 word = S[w * kFold + j];
        const float f[4] = {word.x, word.y, word.z, word.w};
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (4 * w + q < NV) val[4 * w + q] = splat2(f[q]);
    }
}

// Two target rows (standard planes), N values from first_plane, packed lane-wise.
template <int N>
LDDMM_D void load_target_pair(const float4* base, long long stride, long long ra, long long rb, int first_plane,
                              f2* out) {
#pragma unroll
    for (int w = 0; w < (N + 3) / 4; ++w) {
        const float4 a = base[(long long)(first_plane + w) * stride + ra];
        const float4 b = base[(long long)(first_plane + w) * stride + rb];
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (w * 4 + i < N) out[w * 4 + i] = pk2(av[i], bv[i]);
    }
}

template <int KIND, int DEG>
LDDMM_D f2 kval2(const unsigned long long* pkd, f2 r2) {
    if constexpr (KIND == KGAUSS) {
        return ex2neg2(r2);
    } else {
        const f2 u = sqrt2(r2);
        const f2 e = ex2neg2(u);
        if constexpr (DEG == 0) return e;
        else return mul2(horner2<DEG>(pkd, u), e);
    }
}

template <int KIND, int QDEG>
LDDMM_D f2 kdiff2(const unsigned long long* pqd, f2 r2) {
    if constexpr (KIND == KGAUSS) {
        return ex2neg2(r2);
    } else {
        const f2 u = sqrt2(r2);
        const f2 e = ex2neg2(u);
        if constexpr (QDEG == 0) return mul2(f2{pqd[0]}, e);
        else return mul2(horner2<QDEG>(pqd, u), e);
    }
}

// SMALL: groups of 64 targets instead of 128, for a few thousand targets or
// fewer, so that the (target group, source chunk) items spread over the SMs.
template <int KIND, int DEG, int D, int DIMB, bool SMALL = false>
struct OpApplyK2 {
    using Real = float;
    static constexpr bool F32 = true;
    static constexpr bool LIST = true;
    static constexpr int TPS = 2;
    static constexpr int R = SMALL ? 2 : 4;
    static constexpr int PP = 1;            // target planes: pos
    static constexpr int NV = D + DIMB;     // source values
    static constexpr int NS = (NV + 3) / 4; // source words
    static constexpr int NOUT = DIMB;
    using Params = KernelParams2;
    using Acc = AccF32C2<DIMB>;
    using Abs = AccAbs2<DIMB>;
    static constexpr int NW = DIMB, NB = DIMB, DOT = 0;   // bounds: the columns
    static LDDMM_D float lgk(const Params& P, float d2) { return lg_factor<KIND, DEG>(P.pkd, d2); }
    struct Tgt {
        f2 x[D];
    };
    struct Src {
        f2 val[NV];
    };
    static LDDMM_D float coord(const Tgt& t, int h, int j) { return j < D ? half2(t.x[j < D ? j : 0], h) : 0.f; }
    static LDDMM_D void lower(const Tgt&, int, const float* a, float, float* lo) {
#pragma unroll
        for (int c = 0; c < DIMB; ++c) lo[c] = a[c];
    }
    static LDDMM_D void upper(const float* lgw, float, float lk, const float*, float* u) {
#pragma unroll
        for (int c = 0; c < DIMB; ++c) u[c] = lgw[c] + lk;
    }
    static LDDMM_D void load_target(const Params& P, long long ra, long long rb, Tgt& t) {
        load_target_pair<D>(P.tgt4, P.tgt_stride, ra, rb, 0, t.x);
    }
    static LDDMM_D void load_source(const float4* S, int j, Src& s) { load_list_source<NV>(S, j, s.val); }
    template <class A>
    static LDDMM_D void pair(const Params& P, const Tgt& t, const Src& s, A& a) {
        f2 r2;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            const f2 dj = sub2(t.x[j], s.val[j]);
            r2 = j == 0 ? mul2(dj, dj) : fma2(dj, dj, r2);
        }
        const f2 k = kval2<KIND, DEG>(P.pkd, r2);
#pragma unroll
        for (int c = 0; c < DIMB; ++c) a.fma(c, k, s.val[D + c]);
    }
};

template <int KIND, int DEG, int D, int W, bool SMALL = false>
struct OpDiffKT2 {
    using Real = float;
    static constexpr bool F32 = true;
    static constexpr bool LIST = true;
    static constexpr int TPS = 2;
    static constexpr int R = SMALL ? 2 : 4;
    static constexpr int PP = 1;
    static constexpr int NV = D + W;
    static constexpr int NS = (NV + 3) / 4;
    static constexpr int NT = 1 + (W + 3) / 4;  // target planes: pos, u values
    static constexpr int MIN_BLOCKS = 3;        // see op_min_blocks
    static constexpr int NOUT = D;
    using Params = KernelParams2;
    using Acc = AccF32C2<D>;
    using Abs = AccAbs2<D>;
    static constexpr int NW = W, NB = D, DOT = W;   // bounds: the components
    static LDDMM_D float lgk(const Params& P, float d2) { return lg_factor<KIND, DEG>(P.pqd, d2); }
    struct Tgt {
        f2 x[D];
        f2 u[W];
    };
    struct Src {
        f2 val[NV];
    };
    static LDDMM_D float coord(const Tgt& t, int h, int j) { return j < D ? half2(t.x[j < D ? j : 0], h) : 0.f; }
    static LDDMM_D float dot_val(const Tgt& t, int h, int w) { return half2(t.u[w], h); }
    static LDDMM_D void lower(const Tgt&, int, const float* a, float norm1, float* lo) {
#pragma unroll
        for (int j = 0; j < D; ++j) lo[j] = norm1 == 0.f ? -1.f : __fdividef(a[j], norm1);
    }
    static LDDMM_D void upper(const float*, float lgv, float lk, const float* lext, float* u) {
#pragma unroll
        for (int j = 0; j < D; ++j) u[j] = lgv + lk + lext[j];
    }
    static LDDMM_D void load_target(const Params& P, long long ra, long long rb, Tgt& t) {
        load_target_pair<D>(P.tgt4, P.tgt_stride, ra, rb, 0, t.x);
        load_target_pair<W>(P.tgt4, P.tgt_stride, ra, rb, 1, t.u);
    }
    static LDDMM_D void load_source(const float4* S, int j, Src& s) { load_list_source<NV>(S, j, s.val); }
    template <class A>
    static LDDMM_D void pair(const Params& P, const Tgt& t, const Src& s, A& a) {
        f2 dx[D], r2;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            dx[j] = sub2(t.x[j], s.val[j]);
            r2 = j == 0 ? mul2(dx[j], dx[j]) : fma2(dx[j], dx[j], r2);
        }
        f2 dot = mul2(t.u[0], s.val[D]);
#pragma unroll
        for (int w = 1; w < W; ++w) dot = fma2(t.u[w], s.val[D + w], dot);
        const f2 g = mul2(kdiff2<KIND, DEG>(P.pqd, r2), dot);
#pragma unroll
        for (int j = 0; j < D; ++j) a.fma(j, g, dx[j]);
    }
};

// Host: duplicated polynomial coefficients for KernelParams2.
inline unsigned long long dup_coeff(double c) {
    const float f = (float)c;
    unsigned int u;
    memcpy(&u, &f, 4);
    return ((unsigned long long)u << 32) | (unsigned long long)u;
}

}  // namespace lddmm
