// Host-side planning, launching and template dispatch for sweep_kernel.
#pragma once
#include <cmath>
#include <type_traits>

#include "host.h"
#include "ops2.cuh"
#include "sweep.cuh"

namespace lddmm {

template <int V>
using IC = std::integral_constant<int, V>;

// Problems with at most this many targets use the SMALL shape of the operators
// that have one (groups of 64 targets: more, smaller items).
#ifndef LDDMM_SMALL_TARGETS
#define LDDMM_SMALL_TARGETS 4096
#endif
constexpr long long kSmallTargets = LDDMM_SMALL_TARGETS;

struct SinglePlan {
    long long n_tpad, m_pad;
    int n_tb, n_folds, split;
    bool seq;   // FP64 sums over few sources: sweep_seq_kernel, coordinates in the x/s frame (kfun.cuh)
    // chunk sums (doubles) of a sweep with an epilogue: none where a group has one chunk
    size_t part_doubles(int nout) const { return split > 1 ? (size_t)split * n_tpad * nout : 0; }
    size_t counters() const { return (size_t)n_tb + 1; }
    // The fold boxes; NULL, which the pack kernels and epilogues understand, where no fold is bounded.
    // (Formed all the same they cost a shot and adjoint of 1,000 / 2,000 points 248 / 291 us
    // instead of 216 / 253.)
    template <class Op>
    float4* take_boxes(Workspace& ws, int unbounded = kBoundFolds) const {
        if (n_folds <= unbounded) return nullptr;
        return ws.take<float4>((size_t)fold_box_words(op_weights<Op>()) * (size_t)(m_pad / kFold));
    }
};

template <class Op>
SinglePlan plan_single(long long n, long long m, int split_cap = 0, bool shared = false) {
    SinglePlan p;
    const long long per_group = op_group<Op>();
    p.n_tb = (int)((n + per_group - 1) / per_group);
    p.n_tpad = (long long)std::max(p.n_tb, 1) * per_group;
    p.n_folds = (int)((m + kFold - 1) / kFold);
    p.m_pad = (long long)std::max(p.n_folds, 1) * kFold;
    const int sms = device_info().sms;
    p.split = choose_split(p.n_tb, p.n_folds, sms, sms * op_min_blocks<Op>(), shared);
    p.seq = sizeof(typename Op::Real) == 8 && p.n_folds <= kSeqFolds;
    if (p.seq) p.split = 1;
    if (split_cap > 0 && p.split > split_cap) p.split = split_cap;
    return p;
}

// Order of the target rows of a sum over its own points (perm NULL: as they lie),
// from 32,768 points on: the five launches (15 us) and a shot's box launch per step
// (3 us) are 1-4% of sums that take 350 us each when nothing is far, and save a
// third where the kernel is narrow (launch_order_rows).
struct OrderRows {
    int *perm = nullptr, *hist = nullptr, *cell = nullptr, *tmp = nullptr;
};
constexpr long long kOrderRowsMin = 32768;
inline OrderRows take_order(Workspace& ws, long long n_pad) {
    OrderRows o;
    o.perm = ws.take<int>(n_pad);
    o.hist = ws.take<int>(2 * kOrderCells + 1);
    o.cell = ws.take<int>(n_pad);
    o.tmp = ws.take<int>(n_pad);
    if (ws.measuring()) o.perm = nullptr;
    return o;
}
inline OrderRows take_order_rows(Workspace& ws, const SinglePlan& pl) {
    if (pl.seq || (long long)pl.n_folds * kFold < kOrderRowsMin) return OrderRows{};
    return take_order(ws, pl.n_tpad);
}
// o.perm of the n rows packed in `planes` (n_pad of them, positions first)
template <class Real>
int launch_order_rows(const OrderRows& o, const float4* planes, long long n, long long n_pad, cudaStream_t st) {
    if (o.perm == nullptr) return LDDMM_OK;
    LDDMM_TRY(cuda_check(cudaMemsetAsync(o.hist, 0, sizeof(int) * (2 * kOrderCells + 1), st), "order memset"));
    const int blocks = grid_for(n_pad);
    int* info = o.hist + 2 * kOrderCells;
    order_extent_kernel<Real><<<(blocks + 7) / 8, 256, 0, st>>>(planes, n_pad, n, info);
    order_cells_kernel<Real><<<blocks, 256, 0, st>>>(planes, n_pad, n, info, o.hist, o.cell);
    order_scan_kernel<<<1, 1024, 0, st>>>(o.hist, info);
    order_scatter_kernel<<<blocks, 256, 0, st>>>(o.cell, n, o.hist + kOrderCells, o.tmp);
    order_rank_kernel<<<blocks, 256, 0, st>>>(o.tmp, o.cell, o.hist, info, n, n_pad, o.perm);
    return cuda_check(cudaGetLastError(), "order rows");
}

// boxes: fold boxes written with the packed sources, or NULL (every fold counts).
// SYM: symmetric sweep over sym_folds own folds (see sweep_kernel<Op, true>).
// self: the first sources are the targets, in their order (a hint: see the far folds).
// Epi: what is done with a group's sums; counters: n_tb + 1 zeros; perm: order of the
// target rows, or NULL (see sweep_kernel).
template <class Op, bool SYM = false, class Epi = EpiNone>
int launch_single(const SinglePlan& pl, long long n, const typename Op::Params& P, const float4* boxes, double* part,
                  cudaStream_t st, int sym_folds = 0, int* counters = nullptr, const Epi& E = Epi(),
                  const int* perm = nullptr, bool self = true) {
    SweepGrid g{};
    g.seg0.n_tgt = (int)n;
    g.seg0.n_folds = pl.n_folds;
    g.seg0.n_tb = pl.n_tb;
    g.seg0.split = pl.split;
    g.seg0.sym_folds = sym_folds;
    g.seg0.perm = perm;
    g.seg0.self = self;
    g.seg0.bound = boxes != nullptr;
    g.nseg = 0;
    g.n_items = pl.n_tb * pl.split;
    if (g.n_items <= 0) return LDDMM_OK;
    if constexpr (sizeof(typename Op::Real) == 8) {
        if (pl.seq) {
            sweep_seq_kernel<Op, Epi><<<pl.n_tb, op_group<Op>(), 0, st>>>(g.seg0, P, part, E);
            return cuda_check(cudaGetLastError(), "sweep launch");
        }
    }
    sweep_kernel<Op, SYM, Epi><<<g.n_items, 32 * kSweepWarps, 0, st>>>(g, P, boxes, part, counters, E);
    return cuda_check(cudaGetLastError(), "sweep launch");
}

// Kernel-dependent prescale of the coordinates, rescaled polynomials, and the
// constant of the derivative sums (see kfun.cuh).
struct KScale {
    double scale;   // coordinate multiplier used when packing
    double pk[5];   // K polynomial in the prescaled variable
    double pq[4];   // K' polynomial in the prescaled variable
    double dscale;  // sum_l K' 2 (x-y) <u,v> = dscale * sum_l F (x'-y') <u,v>
};

// base2: the frame of the sweep kernels; otherwise x/s (see kfun.cuh).
inline KScale kernel_scale(int kind, int order, double sigma, bool base2, bool exact_tables = false) {
    KScale k{};
    double P[5], Q[4], Rr[3];
    laplacian_tables(order, P, Q, Rr, exact_tables);
    const double L = 1.4426950408889634;  // log2(e)
    if (base2) {
        k.scale = (kind == KGAUSS) ? std::sqrt(0.5 * L) / sigma : L / sigma;
        double Lj = 1.0;
        for (int j = 0; j < 5; ++j) {
            k.pk[j] = P[j] / Lj;
            if (j < 4) k.pq[j] = Q[j] / Lj;
            Lj *= L;
        }
    } else {
        k.scale = 1.0 / sigma;
        for (int j = 0; j < 5; ++j) k.pk[j] = P[j];
        for (int j = 0; j < 4; ++j) k.pq[j] = Q[j];
    }
    k.dscale = -1.0 / (sigma * sigma * k.scale);
    return k;
}

// kernel polynomials into either parameter block
inline void set_poly(KernelParamsBase<double>& P, const KScale& ks) {
    for (int j = 0; j < 5; ++j) P.pk[j] = ks.pk[j];
    for (int j = 0; j < 4; ++j) P.pq[j] = ks.pq[j];
}
inline void set_poly(KernelParamsBase<float>& P, const KScale& ks) {
    for (int j = 0; j < 5; ++j) P.pk[j] = (float)ks.pk[j];
    for (int j = 0; j < 4; ++j) P.pq[j] = (float)ks.pq[j];
}
inline void set_poly(KernelParams2& P, const KScale& ks) {
    for (int j = 0; j < 5; ++j) P.pkd[j] = dup_coeff(ks.pk[j]);
    for (int j = 0; j < 4; ++j) P.pqd[j] = dup_coeff(ks.pq[j]);
}

// order > 4: Gaussian; otherwise Laplacian with polynomial degree = order (K)
template <class F>
int dispatch_kind_p(int order, F&& f) {
    switch (order) {
        case 0: return f(IC<KLAP>{}, IC<0>{});
        case 1: return f(IC<KLAP>{}, IC<1>{});
        case 2: return f(IC<KLAP>{}, IC<2>{});
        case 3: return f(IC<KLAP>{}, IC<3>{});
        case 4: return f(IC<KLAP>{}, IC<4>{});
        default: return f(IC<KGAUSS>{}, IC<0>{});
    }
}

// derivative: polynomial degree = order - 1 (order 0 is rejected earlier)
template <class F>
int dispatch_kind_q(int order, F&& f) {
    switch (order) {
        case 1: return f(IC<KLAP>{}, IC<0>{});
        case 2: return f(IC<KLAP>{}, IC<1>{});
        case 3: return f(IC<KLAP>{}, IC<2>{});
        case 4: return f(IC<KLAP>{}, IC<3>{});
        default: return f(IC<KGAUSS>{}, IC<0>{});
    }
}

template <class F>
int dispatch_d(int d, F&& f) {
    if (d <= 2) return f(IC<2>{});
    return f(IC<3>{});
}

template <class F>
int dispatch_dimb(int b, F&& f) {
    switch (b) {
        case 1: return f(IC<1>{});
        case 2: return f(IC<2>{});
        case 3: return f(IC<3>{});
        default: return f(IC<4>{});
    }
}

// inner-product widths built: 1,2,3,4,6,8,9,12 (others padded with zeros)
template <class F>
int dispatch_w(int w, F&& f) {
    if (w <= 1) return f(IC<1>{});
    if (w <= 2) return f(IC<2>{});
    if (w <= 3) return f(IC<3>{});
    if (w <= 4) return f(IC<4>{});
    if (w <= 6) return f(IC<6>{});
    if (w <= 8) return f(IC<8>{});
    if (w <= 9) return f(IC<9>{});
    return f(IC<12>{});
}


}  // namespace lddmm
