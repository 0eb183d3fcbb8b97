// Generic N-body sweep over (target group, source chunk) items.
//
// A block owns GT = 32*R targets (R per thread, kept in registers; all four warps
// hold the same targets) and one chunk of the source range.  Sources are
// handled in folds of 32 consecutive records (NS 16-byte words each, packed
// structure-of-arrays in global memory, see Op::Src).  The 4 * split warps
// that share a target group take every (4 * split)-th fold each, so that the
// folds a group needs (neighbours in memory, when the order of the points
// follows the shape) spread evenly over them.  A warp streams its folds
// through its own cp.async ring: it waits for nobody but itself
// (`__syncwarp`), every lane reads the same record (shared-memory broadcast).
// One fold is 4096 pairs against 1-2 KB from L2, about 5 bytes per clock and SM,
// so sharing a tile between the warps would save nothing that counts.
//
// Per-target accumulators: FP32 partials over the 32 sources of a fold, in
// order, folded into a TwoSum-compensated (sum, err) pair (FP32 ops), or plain
// FP64 sums.  The block adds its warps in order and writes doubles into
//   part[(seg.part + chunk * seg.n_tb * GT + tb * GT + t) * Op::NOUT + c]
// The block of a group that finishes last adds the chunks in their order and
// hands the group's sums to the epilogue Epi (which scales and writes them, or
// takes the Euler step and packs the next sweep's records), so results do not
// depend on scheduling.  The groups' counters start at zero and are left at
// zero.  A separate combine launch per sweep cost 4-10 us of a shot's step at a
// few thousand points (13 blocks, each thread adding its row's chunks one after
// the other).  EpiNone leaves the chunk sums in `part`, chunk by chunk with seg.n_tgt
// rows each.
//
// Far folds (operators with Op::lgk, seg.bound: more than kBoundFolds folds).  The pack
// kernels leave for each fold its bounding box and, by weight column, log2 of the sum of
// its weights.  With the box of the target group these bound what a fold can add
// to an output of any target of the group, U = W_F K(dmin), times max |x_j - y_j| where
// the term carries x - y and |u_k|_1 where it carries <u_k, v_l>.  What the outputs
// hold at least is measured: each warp adds up the absolute terms of all targets of the
// group over eight records of one fold, and L, by output, is the least over the targets
// (per unit of |u_k|_1), of the warps the best.  A fold with
//   U <= L 2^-MARGIN / (number of folds)   for every output
// is passed over: all such folds together stay below 2^-MARGIN of the sum of absolute
// terms of every output of every target, MARGIN = 36 for FP32 pairs (whose own rounding
// is 2^-22 to 2^-24 of it) and 58 for FP64 (2^-53).  A bound by boxes alone would not do:
// near records may add nothing to an output, because they coincide with the target,
// weigh in other columns or are orthogonal to u_k.  The test is done in log2, so it holds
// as well for targets far from every source, where the whole sum is tiny.  A fold with a
// non-finite coordinate or value is never passed over, nor is any by a group with a
// non-finite target; nor where L is 0 or overflows.  A lane tests one fold, a warp 32 at
// a time.
// Measured against the sweep over every pair (B200): FP32c varifold gradient of a
// 20,480-cell sphere at sigma 0.1 0.97 -> 0.41 ms, its FP64 value 1.63 -> 0.58 ms, the
// value of 98,000 cells at sigma 0.05 6.2 -> 1.6 ms.  Where no fold is far it costs 5% of
// a shot and adjoint of 12,300 points (1.8 -> 1.9 ms), less of longer sweeps.
//
// perm (SegDesc): the target rows in an order that puts neighbours into the same
// group (launch_order_rows, pack.cuh).  The sum of a target does not depend on
// its group, but the group's box does: 128 consecutive vertices of a subdivided
// mesh are strung out along its coarser edges.
//
// SYM (symmetric sums, used for energies <S,S> - 2 <S,T> whose summand is
// symmetric in the target and the source): the first seg.sym_folds folds hold
// the targets' own records in target order.  A group skips those of its own
// records that precede it, counts its diagonal folds once and the later ones
// twice (per-fold weight applied to the FP32 partial, exact for 1 and 2), so
// each unordered pair is evaluated once: the per-target partial sums are no
// longer the per-target sums, their weighted total is.
#pragma once
#include <cfloat>
#include <type_traits>

#include "common.cuh"

namespace lddmm {

constexpr int kSweepWarps = 4;     // warps of a sweep block
constexpr int kFold = 32;          // source records per fold

template <class Real>
struct Traits;
template <>
struct Traits<float> {
    static constexpr int PER_WORD = 4;  // values per 16-byte word
};
template <>
struct Traits<double> {
    static constexpr int PER_WORD = 2;
};

template <class Real>
LDDMM_D Real word_get(const float4* w, int i) {
    if constexpr (sizeof(Real) == 4) {
        const float* f = reinterpret_cast<const float*>(w);
        return f[i];
    } else {
        const double* f = reinterpret_cast<const double*>(w);
        return f[i];
    }
}

// Reads `n` consecutive values starting at value index 0 of a record that is
// spread over planes: value i lives in plane (first_plane + i / PER_WORD).
template <class Real, int N>
LDDMM_D void load_vals(const float4* base, long long stride, long long row, int first_plane, Real* out) {
    constexpr int PW = Traits<Real>::PER_WORD;
#pragma unroll
    for (int w = 0; w < (N + PW - 1) / PW; ++w) {
        const float4 word = base[(long long)(first_plane + w) * stride + row];
#pragma unroll
        for (int i = 0; i < PW; ++i)
            if (w * PW + i < N) out[w * PW + i] = word_get<Real>(&word, i);
    }
}

// smem version: plane p of record j of a fold at S[p*kFold + j]
template <class Real, int N>
LDDMM_D void load_vals_smem(const float4* S, int j, int first_plane, Real* out) {
    constexpr int PW = Traits<Real>::PER_WORD;
#pragma unroll
    for (int w = 0; w < (N + PW - 1) / PW; ++w) {
        const float4 word = S[(first_plane + w) * kFold + j];
#pragma unroll
        for (int i = 0; i < PW; ++i)
            if (w * PW + i < N) out[w * PW + i] = word_get<Real>(&word, i);
    }
}

// An operator may accumulate some outputs scaled by a power of two (cheaper per
// pair); Op::out_scale(c) is then the exact factor applied when they are written.
template <class Op, class = void>
struct op_has_out_scale : std::false_type {};
template <class Op>
struct op_has_out_scale<Op, std::void_t<decltype(Op::out_scale(0))>> : std::true_type {};

// An operator may name the resident blocks per SM that its register budget is cut for.
template <class Op, class = void>
struct op_has_min_blocks : std::false_type {};
template <class Op>
struct op_has_min_blocks<Op, std::void_t<decltype(Op::MIN_BLOCKS)>> : std::true_type {};

// Resident blocks per SM and the unrolling of the source loop.  Measured at
// n = m = 131,072 (FP32) and 32,768 (FP64), 1e12 pairs/s:
//   FP32, 8 / 16 / 32 sources unrolled, 128 registers (4 blocks):
//     Gaussian applyK 2.93 / 3.07 / 3.07, Laplacian 1.97 / 2.00 / 2.02,
//     adjoint 1.66 / 1.71 / 1.73, current gradient 1.63 / 1.62 / 1.66
//   gradient sums with 168 registers (3 blocks), 32 sources: Gaussian 2.09 ->
//     2.18, Laplacian 1.67 -> 1.72, adjoint 1.73 -> 1.74
//   FP64, 8 / 16 / 32 sources: applyK 0.646 / 0.658 / 0.653, varifold gradient
//     0.424 / 0.428 / 0.333
//   FP64 Laplacian, whose square roots each carry a rare branch, 2 / 4 / 8 / 16 sources
//     at 40,000: applyK 0.323 / 0.327 / 0.325 / 0.278, applyDiffKT 0.306 / 0.308 /
//     0.305 / 0.255, divergence 0.348 / 0.348 / 0.320 / 0.222 (5 to 8 blocks: less)
// Operators with many outputs or wide records keep 168 registers as well.
template <class Op>
constexpr int op_min_blocks() {
    if constexpr (op_has_min_blocks<Op>::value) return Op::MIN_BLOCKS;
    else if constexpr (sizeof(typename Op::Real) == 4) return Op::NOUT * Op::R > 24 || Op::NS > 6 ? 3 : 4;
    else return Op::NOUT > 4 || Op::NS > 5 ? 3 : 4;
}
template <class Op>
constexpr int op_unroll() {
    if constexpr (sizeof(typename Op::Real) == 4) return kFold;
    else return Op::FAMILY == KLAP ? 4 : kFold / 2;
}

// Operators that can pass over far folds.  They give, with h the half of a packed slot:
//   NW               weight columns of a source record that bound its terms
//   NB               bounds: what a fold adds is compared bound by bound
//   coord(t, h, j)   packed coordinate j of target t
//   DOT, dot_val     columns of the inner product <u_k, v_l> in some terms (0: none), u_k
//   lgk(P, d2)       log2 of the kernel factor at a squared distance (falls with it)
//   lower(t, h, a, norm1, lo)   what target t's sums hold at least, one value per bound,
//                    from a, its sums of absolute terms over some records; per unit of
//                    norm1 = |u_k|_1 where the terms carry <u_k, v_l>; -1: any fold may go
//   upper(lgw, lgv, lk, lext, u)  log2 of what a fold adds to any target, per bound:
//                    lgw its weights by column, lgv of the inner product per unit of
//                    norm1, lk of the kernel factor, lext of |x_j - y_j|
template <class Op, class = void>
struct op_culls : std::false_type {};
template <class Op>
struct op_culls<Op, std::void_t<decltype(&Op::lgk)>> : std::true_type {};
template <class Op>
constexpr int op_weights() {
    if constexpr (op_culls<Op>::value) return Op::NW;
    else return 0;
}

// Up to this many folds (6,144 sources) a sweep is so short that bounding its folds costs
// what it saves; FP32 shots, adjoints and varifold gradients of one problem, a wave or two
// of blocks, up to twice as many (segments of a ragged launch have the others beside them).
// B200, every fold / bounded, us, sigma 0.05 / 0.1 (0.12 of the shots) / 0.2:
//   shot and adjoint of ten steps, FP32, 8,000 points of a sphere 872 / 874 / 875 and
//     909 / 959 / 965, 10,242 points 1344 / 1345 / 1345 and 1284 / 1411 / 1430, 12,000 points
//     1793 / 1791 / 1795 and 1685 / 1884 / 1891
//   varifold gradient, FP32, 3,920 cells 82 / 82 / 82 and 84 / 86 / 86, 5,120 cells
//     100 / 100 / 100 and 97 / 105 / 105, 5,831 cells 117 / 117 / 117 and 115 / 120 / 122
//   varifold value and gradient, FP64, 5,120 cells 150 / 150 / 151 and 106 / 129 / 154,
//     186 / 186 / 186 and 121 / 172 / 194; current gradient, FP32, 84 / 84 and 63 / 71
constexpr int kBoundFolds = 192, kBoundFoldsPacked = 384;

// float4 words of a fold's box: (lo, lgw[0]), (hi, lgw[1]), (lgw[2..5]), ...
constexpr __host__ __device__ int fold_box_words(int nw) { return 2 + (nw > 2 ? (nw + 1) / 4 : 0); }

// log2 of a sum of n values at most, per value
constexpr LDDMM_D float lg_columns(int n) { return n <= 1 ? 0.f : n <= 2 ? 1.f : n <= 4 ? 2.f : n <= 8 ? 3.f : 4.f; }

// Targets of one group.
template <class Op>
constexpr int op_group() { return 32 * Op::R; }

// Squared distances between two boxes: the smallest and the largest, and the largest
// |x_j - y_j|, with slack for the rounding of the pairs' own distances.
struct Box {
    float lo[3], hi[3];
};
LDDMM_D void box_dist2(const Box& a, const float4 lo, const float4 hi, float& dmin2, float& dmax2, float (&ext)[3]) {
    const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
    float mn = 0.f, mx = 0.f;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const float g = fmaxf(0.f, fmaxf(l[j] - a.hi[j], a.lo[j] - h[j]));
        const float f = fmaxf(h[j] - a.lo[j], a.hi[j] - l[j]);
        mn = fmaf(g, g, mn);
        mx = fmaf(f, f, mx);
        ext[j] = f * (1.f + 1.f / 65536.f);
    }
    dmin2 = mn * (1.f - 1.f / 65536.f);
    dmax2 = mx * (1.f + 1.f / 65536.f);
}

LDDMM_D float warp_min(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
LDDMM_D float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

LDDMM_D float lg_float(float v) { return log2f(v); }
LDDMM_D float lg_float(double v) {   // (log2 of the FP32 part and the exponent: a few 2^-24)
    if (!(v > 0.0)) return -INFINITY;
    if (!(v < INFINITY)) return (float)v;
    int e;
    const double m = frexp(v, &e);
    return log2f((float)m) + (float)e;
}

// The box of a fold of packed source records and log2 of the sums of its weights by
// column (see fold_box_words).  Called by whole warps, lane i holding record `row` = 32
// fold + i; `valid`: a real record (padding has none), p its packed position, w[0..nw)
// its values (nw <= NW).  A non-finite value makes all lgw +inf: such a fold is never
// passed over.
template <class Real, int NW>
LDDMM_D void store_fold_box(float4* boxes, long long row, bool valid, const Real* p, const Real* w, int nw) {
    constexpr int WORDS = fold_box_words(NW);
    float lo[3], hi[3], lg[4 * WORDS - 6];
    bool bad = false;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        if constexpr (sizeof(Real) == 4) {
            lo[j] = hi[j] = p[j];
        } else {
            lo[j] = __double2float_rd(p[j]);
            hi[j] = __double2float_ru(p[j]);
        }
        bad = bad || !(fabsf(lo[j]) < INFINITY) || !(fabsf(hi[j]) < INFINITY);
        lo[j] = warp_min(valid ? lo[j] : INFINITY);
        hi[j] = warp_max(valid ? hi[j] : -INFINITY);
    }
#pragma unroll
    for (int c = 0; c < 4 * WORDS - 6; ++c) {
        lg[c] = -INFINITY;
        if (c < NW && c < nw) {
            const Real v = w[c] < (Real)0 ? -w[c] : w[c];
            bad = bad || !(v < (Real)INFINITY);
            Real sum = valid ? v : (Real)0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            lg[c] = lg_float(sum);
        }
    }
    const bool any = __any_sync(0xffffffffu, valid && bad);
    if ((threadIdx.x & 31) == 0) {
        const int words = fold_box_words(nw);
        float4* o = boxes + words * (row / kFold);
#pragma unroll
        for (int c = 0; c < 4 * WORDS - 6; ++c) lg[c] = any ? INFINITY : lg[c];
        o[0] = make_float4(lo[0], lo[1], lo[2], lg[0]);
        o[1] = make_float4(hi[0], hi[1], hi[2], lg[1]);
#pragma unroll
        for (int k = 2; k < WORDS; ++k)
            if (k < words) o[k] = make_float4(lg[4 * k - 6], lg[4 * k - 5], lg[4 * k - 4], lg[4 * k - 3]);
    }
}

// Whether this block is the last of `total` to come here (all threads ask; what
// the others wrote before is visible to the last one).  The counter goes back to
// zero.
LDDMM_D bool last_block(int* counter, int total) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(counter, 1) == total - 1;
        if (last) *counter = 0;
    }
    __syncthreads();
    const bool r = last != 0;
    __threadfence();
    return r;
}

// Sum over the block in a fixed tree; every thread gets it.
LDDMM_D double block_sum_all(double v) {
    __shared__ double ws[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) r += ws[w];
    __syncthreads();
    return r;
}

// Epilogues: run() is called by all threads of a group's last block with the
// group's sums red[r * NOUT + c], r < GT; sum r belongs to the segment's row
// srow[r] where that is below seg.n_tgt.
struct EpiNone {
    static constexpr bool NONE = true;
};

// f[row, col0 + c] = scale * sum, c < ncols
struct EpiSum {
    static constexpr bool NONE = false;
    double* f;
    long long ld;
    int col0, ncols;
    double scale;
    template <int GT, int NOUT>
    LDDMM_D void run(const SegDesc& sg, int, const int* srow, const double* red) const {
        for (int i = threadIdx.x; i < GT * ncols; i += blockDim.x) {
            const int r = i / ncols, c = i - r * ncols, row = srow[r];
            if (row < sg.n_tgt) f[row * ld + col0 + c] = scale * red[r * NOUT + c];
        }
    }
};

template <class Op, bool SYM, class Epi>
__global__ void __launch_bounds__(32 * kSweepWarps, op_min_blocks<Op>())
    sweep_kernel(const SweepGrid grid, const typename Op::Params P, const float4* __restrict__ boxes, double* part,
                 int* counters, const Epi E) {
    constexpr int R = Op::R, TPS = Op::TPS, NS = Op::NS, NOUT = Op::NOUT, GT = op_group<Op>();
    constexpr int STAGE = NS * kFold;   // 16-byte words of one fold
    constexpr int STAGES = NS > 6 ? 2 : 3;   // folds of a warp's ring (at most 48 KB for the block)
    constexpr int RING = kSweepWarps * STAGES * STAGE;
    constexpr int RED = (GT * NOUT * 8 + 15) / 16;
    __shared__ __align__(16) float4 smem[RING > RED ? RING : RED];
    __shared__ Box wbox;                                             // the group's box
    __shared__ float sthr[kSweepWarps][8], sthr_w[kSweepWarps][8];   // log2 of what a fold may add, by bound
    __shared__ unsigned slive_w[kSweepWarps];

    const int item = blockIdx.x;
    const SegDesc sg = find_segment(grid, item);
    const int local = item - sg.item0;
    const int tb = local / sg.split;
    const int chunk = local - tb * sg.split;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    // targets of this lane: rows r*32 + lane of the group (rows are padded); an
    // operator with TPS == 2 keeps two of them per slot (packed FP32 pairs)
    constexpr int SLOTS = R / TPS;
    static_assert(R % TPS == 0, "R must be a multiple of TPS");
    __shared__ int srow[GT];
    typename Op::Tgt tg[SLOTS];
    unsigned valid = 0;   // which of the rows are targets
    int row[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int r = tb * GT + q * 32 + lane;
        row[q] = sg.perm != nullptr ? sg.perm[r] : r;
        if (warp == 0) srow[q * 32 + lane] = row[q];
        if (row[q] < sg.n_tgt) valid |= 1u << q;
    }
    const int n_folds = sg.n_folds;

    // source words: Op lays a record out as NS planes of 16-byte words, plane
    // p of record j at P.src4[p * P.src_stride + j]; a fold's stage is plane-major
    float4* ring = smem + warp * STAGES * STAGE;
    auto load_fold = [&](int f, int st) {
        if (f >= 0) {
            const float4* g = P.src4 + sg.src + (long long)f * kFold + lane;
#pragma unroll
            for (int w = 0; w < NS; ++w) cp_async16(ring + st * STAGE + w * kFold + lane, g + (long long)w * P.src_stride);
        }
        cp_async_commit();
    };

    // far folds: a fold of the group's own rows, another one for each warp where it has as many
    const bool bounded = op_culls<Op>::value && sg.bound;
    int own_fold = -1;
    if (bounded && sg.self) {
        int own = -1;
#pragma unroll
        for (int q = 0; q < R; ++q)
            if (q == warp % R && (valid & (1u << q))) own = row[q];
        own = __shfl_sync(0xffffffffu, own, warp / R * 16 % 32);
        if (own < 0) own = __shfl_sync(0xffffffffu, row[0], 0);   // (a group has one target at least)
        own_fold = min(own / kFold, n_folds - 1);
        load_fold(own_fold, 0);
    }
#pragma unroll
    for (int q = 0; q < SLOTS; ++q) {
        if constexpr (TPS == 1) Op::load_target(P, sg.tgt + row[q], tg[q]);
        else Op::load_target(P, sg.tgt + row[q * TPS], sg.tgt + row[q * TPS + 1], tg[q]);
    }
    typename Op::Acc acc[SLOTS];
#pragma unroll
    for (int q = 0; q < SLOTS; ++q) acc[q].zero();

    int f_lo = 0, diag_hi = 0;   // SYM: own folds at or after diag_hi (and before sym_folds) count twice
    if constexpr (SYM) {
        f_lo = min(tb * (GT / kFold), sg.sym_folds);
        diag_hi = tb * (GT / kFold) + GT / kFold;
    }

    // the group's box and, by bound, what a fold may add at most to be passed over
    bool cull = false;
    constexpr int BW = fold_box_words(op_weights<Op>());
    const float4* fbox = nullptr;
    if constexpr (op_culls<Op>::value) {
        if (bounded) {
            fbox = boxes + BW * (sg.src / kFold);
            using Real = typename Op::Real;
            constexpr int NB = Op::NB;
            // every warp holds all targets of the group: the box needs no exchange
            Box wb{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
            bool bad = false;
#pragma unroll
            for (int q = 0; q < R; ++q) {
                if (!(valid & (1u << q))) continue;
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const Real x = Op::coord(tg[q / TPS], q % TPS, j);
                    float l, h;
                    if constexpr (sizeof(Real) == 4) {
                        l = h = x;
                    } else {
                        l = __double2float_rd(x);
                        h = __double2float_ru(x);
                    }
                    bad = bad || !(fabsf(l) < INFINITY) || !(fabsf(h) < INFINITY);
                    wb.lo[j] = fminf(wb.lo[j], l);
                    wb.hi[j] = fmaxf(wb.hi[j], h);
                }
            }
            cull = !__any_sync(0xffffffffu, bad);
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                wb.lo[j] = warp_min(wb.lo[j]);
                wb.hi[j] = warp_max(wb.hi[j]);
            }
            // a fold whose records the targets' sums are compared with: of the group's own rows, or else
            // the one that adds most by its box, of 512 spread over the range (each warp its share)
            int bf = own_fold;
            if (!sg.self) {
                constexpr int PER = 4, LANES = 32 * kSweepWarps;
                const int step = (n_folds + PER * LANES - 1) / (PER * LANES);
                float best = -INFINITY;
                float4 bx[PER][BW];
                int fs[PER];
#pragma unroll
                for (int k = 0; k < PER; ++k) {   // all loads before the first use
                    fs[k] = min((k * LANES + (int)threadIdx.x) * step, n_folds - 1);
#pragma unroll
                    for (int w = 0; w < BW; ++w) bx[k][w] = fbox[BW * fs[k] + w];
                }
#pragma unroll
                for (int k = 0; k < PER; ++k) {
                    float d0, d1, ext[3];
                    box_dist2(wb, bx[k][0], bx[k][1], d0, d1, ext);
                    float lw = fmaxf(bx[k][0].w, bx[k][1].w);
#pragma unroll
                    for (int w = 2; w < BW; ++w)
                        lw = fmaxf(lw, fmaxf(fmaxf(bx[k][w].x, bx[k][w].y), fmaxf(bx[k][w].z, bx[k][w].w)));
                    const float v = lw + Op::lgk(P, d1);
                    if (lw < INFINITY && v > best) {
                        best = v;
                        bf = fs[k];
                    }
                }
                const float top = warp_max(best);
                bf = __reduce_max_sync(0xffffffffu, best == top ? bf : -1);
                if (bf >= 0) load_fold(bf, 0);
            }
            // the targets' sums of absolute terms over a quarter of its records: what their sums over all
            // sources hold at least; the least over the group, 0 where nothing may be passed over
            Real least[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b) least[b] = (Real)INFINITY;
            unsigned live = 0;
            if (bf >= 0) {
                cp_async_wait<0>();
                __syncwarp();
                typename Op::Abs sum[SLOTS];
#pragma unroll
                for (int q = 0; q < SLOTS; ++q) sum[q].zero();
#pragma unroll 2
                for (int j = warp; j < kFold; j += kSweepWarps) {
                    typename Op::Src s;
                    Op::load_source(ring, j, s);
#pragma unroll
                    for (int q = 0; q < SLOTS; ++q) Op::pair(P, tg[q], s, sum[q]);
                }
                __syncwarp();
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    if (!(valid & (1u << q))) continue;
                    Real a[NOUT], lo[NB], norm1 = 0;
#pragma unroll
                    for (int c = 0; c < NOUT; ++c) {
                        a[c] = sum[q / TPS].value(c, q % TPS);
                        if constexpr (op_has_out_scale<Op>::value) a[c] *= (Real)Op::out_scale(c);
                    }
                    if constexpr (Op::DOT > 0) {
#pragma unroll
                        for (int w = 0; w < Op::DOT; ++w) {
                            const Real u = Op::dot_val(tg[q / TPS], q % TPS, w);
                            norm1 += u < (Real)0 ? -u : u;
                            if (u != (Real)0) live |= 1u << w;
                        }
                    }
                    Op::lower(tg[q / TPS], q % TPS, a, norm1, lo);
#pragma unroll
                    for (int b = 0; b < NB; ++b) {
                        if (lo[b] == (Real)-1) continue;
                        if (!(lo[b] < least[b])) lo[b] = lo[b] < (Real)INFINITY ? least[b] : (Real)0;
                        least[b] = lo[b];
                    }
                }
            }
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                float l = bf >= 0 ? lg_float(least[b]) : -INFINITY;
                l = warp_min(l);
                if (lane == 0) sthr_w[warp][b] = l;
            }
            if constexpr (Op::DOT > 0) {
                live = __reduce_or_sync(0xffffffffu, live);   // (the same in every warp that has a fold)
                if (lane == 0) slive_w[warp] = live;
            }
            if (threadIdx.x == 0) wbox = wb;
            __syncthreads();
            if (lane < NB) {
                float l = sthr_w[0][lane];
                for (int w = 1; w < kSweepWarps; ++w) l = fmaxf(l, sthr_w[w][lane]);
                constexpr float kMargin = sizeof(Real) == 4 ? 36.1f : 58.1f;
                sthr[warp][lane] = fminf(l, FLT_MAX) - kMargin - log2f((float)n_folds) - (SYM ? 1.f : 0.f);
            }
            __syncwarp();
        }
    }
    unsigned live = 0;   // columns of the inner product that some target of the group has
    if constexpr (op_culls<Op>::value)
        if constexpr (Op::DOT > 0)
            if (cull)
                for (int w = 0; w < kSweepWarps; ++w) live |= slive_w[w];

    // this warp's folds: f_lo + c, f_lo + c + C, ...; next() gives the next one that counts, -1 after the last
    const int C = sg.split * kSweepWarps;
    int f_base = f_lo + chunk * kSweepWarps + warp, f_cur = 0;
    unsigned f_mask = 0;
    auto next = [&]() -> int {
        while (f_mask == 0) {
            if (f_base >= n_folds) return -1;
            const long long f = (long long)f_base + (long long)lane * C;
            bool act = f < n_folds;
            if constexpr (op_culls<Op>::value) {
                if (cull && act) {
                    float d0, d1, ext[3], lgw[4 * BW - 6], u[Op::NB];
                    const float4 bl = fbox[BW * f], bh = fbox[BW * f + 1];
                    box_dist2(wbox, bl, bh, d0, d1, ext);
                    lgw[0] = bl.w;
                    lgw[1] = bh.w;
#pragma unroll
                    for (int k = 2; k < BW; ++k) {
                        const float4 q = fbox[BW * f + k];
                        lgw[4 * k - 6] = q.x, lgw[4 * k - 5] = q.y, lgw[4 * k - 4] = q.z, lgw[4 * k - 3] = q.w;
                    }
                    float lgv = -INFINITY;   // sum over the records of max |v_w| over the columns in use
#pragma unroll
                    for (int w = 0; w < Op::DOT; ++w)
                        if (live & (1u << w)) lgv = fmaxf(lgv, lgw[w]);
                    lgv += lg_columns(Op::DOT);
#pragma unroll
                    for (int j = 0; j < 3; ++j) ext[j] = __log2f(ext[j]);
                    Op::upper(lgw, lgv, Op::lgk(P, d0), ext, u);
                    act = !(lgw[0] < INFINITY);
#pragma unroll
                    for (int b = 0; b < Op::NB; ++b) act = act || !(u[b] <= sthr[warp][b]);
                }
            }
            f_mask = __ballot_sync(0xffffffffu, act);
            f_cur = f_base;
            f_base = (int)min((long long)f_base + 32LL * C, (long long)n_folds);
        }
        const int b = __ffs(f_mask) - 1;
        f_mask &= f_mask - 1;
        return f_cur + b * C;
    };

    int fa = next(), fb = -1;   // the fold to do, and (three stages) the one after it
    load_fold(fa, 0);
    if constexpr (STAGES == 3) {
        if (fa >= 0) fb = next();
        load_fold(fb, 1);
    }
    int st = 0;
    while (fa >= 0) {
        const int fn = (STAGES == 2 || fb >= 0) ? next() : -1;
        load_fold(fn, st >= 1 ? st - 1 : STAGES - 1);
        cp_async_wait<STAGES - 1>();
        __syncwarp();
        const float4* S = ring + st * STAGE;
#pragma unroll
        for (int q = 0; q < SLOTS; ++q) acc[q].begin_fold();
#pragma unroll op_unroll<Op>()
        for (int j = 0; j < kFold; ++j) {
            typename Op::Src s;
            Op::load_source(S, j, s);
#pragma unroll
            for (int q = 0; q < SLOTS; ++q) Op::pair(P, tg[q], s, acc[q]);
        }
#pragma unroll
        for (int q = 0; q < SLOTS; ++q) {
            if constexpr (SYM) acc[q].end_fold_w(fa >= diag_hi && fa < sg.sym_folds ? 2.f : 1.f);
            else acc[q].end_fold();
        }
        __syncwarp();
        fa = STAGES == 3 ? fb : fn;
        fb = fn;
        st = st == STAGES - 1 ? 0 : st + 1;
    }
    cp_async_wait<0>();
    __syncthreads();

    // add the warps in order, then one coalesced row block of doubles
    double* red = reinterpret_cast<double*>(smem);
    for (int w = 0; w < kSweepWarps; ++w) {
        if (warp == w) {
#pragma unroll
            for (int q = 0; q < SLOTS; ++q) {
#pragma unroll
                for (int l = 0; l < TPS; ++l) {
                    const int t = (q * TPS + l) * 32 + lane;
#pragma unroll
                    for (int c = 0; c < NOUT; ++c) {
                        double v;
                        if constexpr (TPS == 1) v = acc[q].value(c);
                        else v = acc[q].value(c, l);
                        if constexpr (op_has_out_scale<Op>::value) v *= Op::out_scale(c);
                        red[t * NOUT + c] = w == 0 ? v : red[t * NOUT + c] + v;
                    }
                }
            }
        }
        __syncthreads();
    }
    if constexpr (Epi::NONE) {
        const int rows = min(GT, sg.n_tgt - tb * GT);   // (targets as they lie)
        double* dst = part + (sg.part + (long long)chunk * sg.n_tgt + (long long)tb * GT) * NOUT;
        for (int i = threadIdx.x; i < rows * NOUT; i += 32 * kSweepWarps) dst[i] = red[i];
    } else {
        if (sg.split > 1) {
            const long long step = (long long)sg.n_tb * GT * NOUT;
            double* p0 = part + (sg.part + (long long)tb * GT) * NOUT;
            for (int i = threadIdx.x; i < GT * NOUT; i += 32 * kSweepWarps) p0[chunk * step + i] = red[i];
            if (!last_block(counters + sg.cnt + tb, sg.split)) return;
            for (int i = threadIdx.x; i < GT * NOUT; i += 32 * kSweepWarps) {
                double v = 0.0;
                for (int k0 = 0; k0 < sg.split; k0 += 16) {   // 16 loads in flight
                    double q[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) q[j] = k0 + j < sg.split ? __ldcg(p0 + (k0 + j) * step + i) : 0.0;
#pragma unroll
                    for (int j = 0; j < 16; ++j) v += q[j];
                }
                red[i] = v;
            }
            __syncthreads();
        }
        E.template run<GT, NOUT>(sg, tb, srow, red);
    }
}

// FP64 sums over at most kSeqFolds folds (384 sources): one thread per target adds all
// sources in their order, as the reference's loop does.  An optimiser run on a few
// hundred points amplifies the last bits of its FP64 sums by 1e7 over 50 iterations, so
// these keep the reference's order to the bit.  A thread's chain of 480 terms takes
// 64-73 us however many targets there are, the split sweep 18 us (64 x 480 points,
// B200), so the line is where the longest such chain was before there was a choice.
constexpr int kSeqFolds = 12;
template <class Op, class Epi>
__global__ void __launch_bounds__(op_group<Op>()) sweep_seq_kernel(const SegDesc sg, const typename Op::Params P,
                                                                   double* part, const Epi E) {
    static_assert(Op::TPS == 1, "unpacked operators");
    constexpr int NS = Op::NS, NOUT = Op::NOUT, GT = op_group<Op>();
    __shared__ __align__(16) float4 S[NS * kFold];
    __shared__ double red[GT * NOUT];
    const int t = blockIdx.x * GT + threadIdx.x;   // rows are padded to whole groups
    typename Op::Tgt tg;
    Op::load_target(P, sg.tgt + t, tg);
    typename Op::Acc acc;
    acc.zero();
    for (int f = 0; f < sg.n_folds; ++f) {
        const float4* g = P.src4 + sg.src + (long long)f * kFold;
        __syncthreads();
        for (int i = threadIdx.x; i < NS * kFold; i += GT) S[i] = g[(long long)(i / kFold) * P.src_stride + i % kFold];
        __syncthreads();
#pragma unroll 4
        for (int j = 0; j < kFold; ++j) {
            typename Op::Src s;
            Op::load_source(S, j, s);
            Op::template pair<true>(P, tg, s, acc);
        }
    }
    if constexpr (Epi::NONE) {
        if (t < sg.n_tgt)
            for (int c = 0; c < NOUT; ++c) part[(sg.part + t) * NOUT + c] = acc.value(c);
    } else {
        __shared__ int srow[GT];
        srow[threadIdx.x] = t;
        for (int c = 0; c < NOUT; ++c) red[threadIdx.x * NOUT + c] = acc.value(c);
        __syncthreads();
        E.template run<GT, NOUT>(sg, blockIdx.x, srow, red);
    }
}

// ---------------------------------------------------------------------------
// Accumulators
// ---------------------------------------------------------------------------
// FP32 partial over FOLD sources + TwoSum-compensated running sum.
template <int N>
struct AccF32C {
    float p[N], s[N], e[N];
    LDDMM_D void zero() {
#pragma unroll
        for (int c = 0; c < N; ++c) s[c] = e[c] = 0.f;
    }
    LDDMM_D void begin_fold() {
#pragma unroll
        for (int c = 0; c < N; ++c) p[c] = 0.f;
    }
    LDDMM_D void end_fold() {
#pragma unroll
        for (int c = 0; c < N; ++c) two_sum_acc(s[c], e[c], p[c]);
    }
    LDDMM_D void end_fold_w(float w) {
#pragma unroll
        for (int c = 0; c < N; ++c) two_sum_acc(s[c], e[c], p[c] * w);
    }
    LDDMM_D void add(int c, float v) { p[c] += v; }
    LDDMM_D void fma(int c, float a, float b) { p[c] = fmaf(a, b, p[c]); }
    LDDMM_D double value(int c) const { return (double)s[c] + (double)e[c]; }
};

// Sums of the terms' absolute values (one target).
template <class Real, int N>
struct AccAbs {
    Real a[N];
    LDDMM_D void zero() {
#pragma unroll
        for (int c = 0; c < N; ++c) a[c] = 0;
    }
    LDDMM_D void add(int c, Real v) { a[c] += v < (Real)0 ? -v : v; }
    LDDMM_D void fma(int c, Real x, Real y) { add(c, x * y); }
    LDDMM_D Real value(int c, int) const { return a[c]; }
};

// Plain FP64 accumulation (the uncompensated FP64 comparator path).
template <int N>
struct AccF64 {
    double s[N];
    LDDMM_D void zero() {
#pragma unroll
        for (int c = 0; c < N; ++c) s[c] = 0.0;
    }
    double m[N];   // running sum at the start of the fold (symmetric sweeps)
    LDDMM_D void begin_fold() {
#pragma unroll
        for (int c = 0; c < N; ++c) m[c] = s[c];
    }
    LDDMM_D void end_fold() {}
    LDDMM_D void end_fold_w(float w) {
        if (w != 1.f)
#pragma unroll
            for (int c = 0; c < N; ++c) s[c] = m[c] + (double)w * (s[c] - m[c]);
    }
    LDDMM_D void add(int c, double v) { s[c] += v; }
    LDDMM_D void fma(int c, double a, double b) { s[c] = fma_rn(a, b, s[c]); }
    LDDMM_D double value(int c) const { return s[c]; }
    static LDDMM_D double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
};

}  // namespace lddmm
