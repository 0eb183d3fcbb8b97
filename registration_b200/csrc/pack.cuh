// Packing kernels (FP64 user arrays -> prescaled FP32/FP64 planes), the packing
// centre, and the order of rows by cells.
#pragma once
#include "common.cuh"
#include "ops.cuh"

namespace lddmm {

// Centre of the bounding box of x (n, d) and y (m, d): center[0..d).  The
// kernels are translation invariant, and packing coordinates relative to this
// centre halves the magnitude (and so the FP32 rounding error) of the packed
// coordinates.
//
// Blocks reduce min / max of order-preserving 64-bit keys of the coordinates
// (exact, so the result does not depend on their order): one block up to
// kBboxOneBlock points (one launch, 3 us; a launch that zeroes atomics and one
// that reads them back cost 2 us each), otherwise a block per 2048 points leaves
// its six keys for a second, one-block launch.  Ragged launches commit with
// atomicMin / atomicMax into their segment's keys.
constexpr long long kBboxOneBlock = 8192;
constexpr int kBboxMaxBlocks = 592;
constexpr int kCenterWords = 4 + 6 * kBboxMaxBlocks;   // doubles: the centre in [0, 4), then the blocks' keys
constexpr long long kKeyMax = 0x7FFFFFFFFFFFFFFFLL;
constexpr long long kKeyMin = -kKeyMax - 1;

// signed-integer order of the keys == numeric order of the doubles (no NaN)
LDDMM_D long long bbox_key(double v) {
    const long long b = __double_as_longlong(v);
    return b >= 0 ? b : (b ^ kKeyMax);
}

LDDMM_D double bbox_val(long long k) { return __longlong_as_double(k >= 0 ? k : (k ^ kKeyMax)); }

// warp + block reduction of per-thread key bounds; thread 0 gets the block's (min in l, max in h)
LDDMM_D void bbox_block_reduce(long long (&l)[3], long long (&h)[3]) {
    __shared__ long long sl[3][32], sh[3][32];
    for (int off = 16; off > 0; off >>= 1)
        for (int j = 0; j < 3; ++j) {
            l[j] = min(l[j], __shfl_down_sync(0xffffffffu, l[j], off));
            h[j] = max(h[j], __shfl_down_sync(0xffffffffu, h[j], off));
        }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0)
        for (int j = 0; j < 3; ++j) {
            sl[j][warp] = l[j];
            sh[j][warp] = h[j];
        }
    __syncthreads();
    if (warp == 0) {
        for (int j = 0; j < 3; ++j) {
            l[j] = lane < nw ? sl[j][lane] : kKeyMax;
            h[j] = lane < nw ? sh[j][lane] : kKeyMin;
        }
        for (int off = 16; off > 0; off >>= 1)
            for (int j = 0; j < 3; ++j) {
                l[j] = min(l[j], __shfl_down_sync(0xffffffffu, l[j], off));
                h[j] = max(h[j], __shfl_down_sync(0xffffffffu, h[j], off));
            }
    }
}

// one atomic per block and component into keys[0..3) (min) and keys[3..6) (max)
LDDMM_D void bbox_block_commit(long long (&l)[3], long long (&h)[3], long long* keys) {
    bbox_block_reduce(l, h);
    if (threadIdx.x == 0)
        for (int j = 0; j < 3; ++j) {
            if (l[j] != kKeyMax) atomicMin(keys + j, l[j]);
            if (h[j] != kKeyMin) atomicMax(keys + 3 + j, h[j]);
        }
}

LDDMM_D void bbox_write_center(const long long (&l)[3], const long long (&h)[3], int d, bool nonempty,
                               double* center) {
    for (int j = 0; j < 3; ++j) center[j] = (j < d && nonempty) ? 0.5 * (bbox_val(l[j]) + bbox_val(h[j])) : 0.0;
}

// gridDim 1: the centre; otherwise each block's keys
static __global__ void bbox_part_kernel(const double* __restrict__ x, long long n, const double* __restrict__ y,
                                        long long m, int d, double* __restrict__ center) {
    long long l[3] = {kKeyMax, kKeyMax, kKeyMax}, h[3] = {kKeyMin, kKeyMin, kKeyMin};
#pragma unroll 4
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n + m;
         i += (long long)gridDim.x * blockDim.x) {
        const double* p = i < n ? x + i * d : y + (i - n) * d;
        for (int j = 0; j < d; ++j) {
            const long long k = bbox_key(p[j]);
            l[j] = min(l[j], k);
            h[j] = max(h[j], k);
        }
    }
    bbox_block_reduce(l, h);
    if (threadIdx.x != 0) return;
    if (gridDim.x == 1) {
        bbox_write_center(l, h, d, n + m > 0, center);
    } else {
        long long* keys = reinterpret_cast<long long*>(center + 4) + 6 * blockIdx.x;
        for (int j = 0; j < 3; ++j) {
            keys[j] = l[j];
            keys[3 + j] = h[j];
        }
    }
}

static __global__ void bbox_finish_kernel(int blocks, int d, double* __restrict__ center) {
    long long l[3] = {kKeyMax, kKeyMax, kKeyMax}, h[3] = {kKeyMin, kKeyMin, kKeyMin};
    const long long* keys = reinterpret_cast<const long long*>(center + 4);
    for (int b = threadIdx.x; b < blocks; b += blockDim.x)
        for (int j = 0; j < 3; ++j) {
            l[j] = min(l[j], keys[6 * b + j]);
            h[j] = max(h[j], keys[6 * b + 3 + j]);
        }
    bbox_block_reduce(l, h);
    if (threadIdx.x == 0) bbox_write_center(l, h, d, true, center);
}

// center: kCenterWords doubles of device memory (see above)
inline void launch_bbox_center(const double* x, long long n, const double* y, long long m, int d, double* center,
                               cudaStream_t st) {
    const long long tot = n + m;
    if (tot <= kBboxOneBlock) {
        bbox_part_kernel<<<1, 1024, 0, st>>>(x, n, y, m, d, center);
        return;
    }
    const int blocks = (int)std::min<long long>(kBboxMaxBlocks, (tot + 2047) / 2048);
    bbox_part_kernel<<<blocks, 256, 0, st>>>(x, n, y, m, d, center);
    bbox_finish_kernel<<<1, 256, 0, st>>>(blocks, d, center);
}

// Gather spec for value planes: value w of row i is src[i*row_stride + off[w]] * mult.
struct Gather {
    const double* src;
    long long row_stride;
    long long off[12];
    int nvals;
    double mult;
};

// Packed row i of a kernel sum: the position (x_i - center) * scale, then the
// gather's values (V of them at most, zero beyond g.nvals).  LIST (packed FP32
// sources, ops2.cuh): one list of D + V values; otherwise the standard planes,
// position first (FP32: one float4 word; FP64: two double2 words).  boxes
// (sources): the fold's box.  Rows >= n are zero.
template <class Real, bool LIST>
LDDMM_D void pack_row(const double* __restrict__ x, long long n, int d, double scale,
                      const double* __restrict__ center, const Gather& g, int D, int V, float4* __restrict__ out,
                      long long stride, long long i, float4* boxes) {
    constexpr int PW = Traits<Real>::PER_WORD;
    Real v[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = 0;
    const int V0 = LIST ? D : 4;   // first value
    if (i < n) {
        for (int j = 0; j < d && j < 3; ++j) v[j] = (Real)((x[i * d + j] - center[j]) * scale);
        for (int q = 0; q < V && q < g.nvals; ++q) v[V0 + q] = (Real)(g.src[i * g.row_stride + g.off[q]] * g.mult);
    }
    const int nwords = LIST ? (D + V + PW - 1) / PW : 4 / PW + (V + PW - 1) / PW;
    for (int k = 0; k < nwords; ++k) {
        float4* dst = out + (long long)k * stride + i;
        if constexpr (sizeof(Real) == 4) *dst = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
        else *reinterpret_cast<double2*>(dst) = make_double2(v[2 * k], v[2 * k + 1]);
    }
    if (boxes != nullptr) {
        const Real p[3] = {v[0], v[1], D > 2 ? v[2] : (Real)0};
        store_fold_box<Real, 12>(boxes, i, i < n, p, v + V0, V);
    }
}

// Targets (standard planes), then sources of a kernel sum, one launch; zeroes the sweep's counters.
template <class Real, bool LIST>
static __global__ void pack_sum_kernel(const double* __restrict__ x, long long n, const Gather gt, int Vt,
                                       float4* __restrict__ tgt, long long n_tpad, const double* __restrict__ y,
                                       long long m, const Gather gs, int D, int Vs, float4* __restrict__ src,
                                       long long m_pad, int d, double scale, const double* __restrict__ center,
                                       float4* __restrict__ boxes, int* __restrict__ counters, int n_counters) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n_tpad + m_pad;
         q += (long long)gridDim.x * blockDim.x) {
        if (q < n_counters) counters[q] = 0;
        if (q < n_tpad)
            pack_row<Real, false>(x, n, d, scale, center, gt, D, Vt, tgt, n_tpad, q, nullptr);
        else
            pack_row<Real, LIST>(y, m, d, scale, center, gs, D, Vs, src, m_pad, q - n_tpad, boxes);
    }
}

// Fold boxes of packed source rows (list records of D + V values, or standard
// planes with V values).
template <class Real, bool LIST>
static __global__ void fold_boxes_kernel(const float4* __restrict__ src, long long m_pad, long long n, int D, int V,
                                         float4* __restrict__ boxes) {
    constexpr int PW = Traits<Real>::PER_WORD;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < m_pad;
         i += (long long)gridDim.x * blockDim.x) {
        Real p[3] = {0, 0, 0}, w[12];
        const int first = LIST ? D : 4, total = first + V;
        for (int k = 0; k * PW < total; ++k) {
            const float4 word = src[(long long)k * m_pad + i];
            for (int q = 0; q < PW; ++q) {
                const int j = k * PW + q;
                const Real v = word_get<Real>(&word, q);
                if (j < 3 && j < D) p[j] = v;
                if (j >= first && j < total) w[j - first] = v;
            }
        }
        store_fold_box<Real, 12>(boxes, i, i < n, p, w, V);
    }
}

// Standard FP64 records in the order of perm, with V values each, and their fold boxes.
static __global__ void permute_records_kernel(const float4* __restrict__ src, const int* __restrict__ perm,
                                              long long m_pad, long long m, int V, float4* __restrict__ out,
                                              float4* __restrict__ boxes) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < m_pad;
         q += (long long)gridDim.x * blockDim.x) {
        const long long i = perm[q];
        double p[4] = {0, 0, 0, 0}, w[12];
        for (int k = 0; k < 2 + (V + 1) / 2; ++k) {
            const float4 word = src[(long long)k * m_pad + i];
            out[(long long)k * m_pad + q] = word;
            for (int h = 0; h < 2; ++h) {
                const double v = word_get<double>(&word, h);
                if (k < 2) p[2 * k + h] = v;
                else if (2 * (k - 2) + h < V) w[2 * (k - 2) + h] = v;
            }
        }
        store_fold_box<double, 12>(boxes, q, i < m, p, w, V);
    }
}

// Order of the target rows by cells of a 32 x 32 x 32 grid over the packed points,
// the cells along a Morton curve, the rows of a cell as they lie: a counting sort
// whose result does not depend on scheduling (counts are whole numbers; the rows
// that the scatter leaves in any order within a cell are ranked by their number).
// Where the points crowd into a few cells (over kOrderCrowd rows in one) the rows
// keep their order.  On a sphere of 40,962 subdivided vertices at sigma 0.05 the
// groups' boxes let a sweep pass over 73% of the pairs instead of 55%.
constexpr int kOrderCells = 32768, kOrderCrowd = 2048;
LDDMM_D unsigned morton_spread(unsigned v) {   // 5 bits to every third
    v = (v | (v << 8)) & 0x0000100Fu;
    v = (v | (v << 4)) & 0x000010C3u;
    return (v | (v << 2)) & 0x00001249u;
}
// info[0] (zero before): bits of the largest finite |coordinate|, the same whatever the blocks' order.
// (One block over all points took 100 us of an FP64 sum of 2,048 x 524,288: 2.07 -> 1.95 ms.)
template <class Real>
static __global__ void __launch_bounds__(256) order_extent_kernel(const float4* __restrict__ tgt, long long stride,
                                                                  long long n, int* __restrict__ info) {
    __shared__ float sm[8];
    float m = 0.f;
#pragma unroll 4
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < n; i += gridDim.x * 256LL) {
        Real x[3];
        load_vals<Real, 3>(tgt, stride, i, 0, x);
        for (int j = 0; j < 3; ++j) {
            const float v = fabsf((float)x[j]);
            if (v < INFINITY) m = fmaxf(m, v);
        }
    }
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) m = fmaxf(m, sm[w]);
        atomicMax(info, __float_as_int(m));
    }
}
template <class Real>
static __global__ void order_cells_kernel(const float4* __restrict__ tgt, long long stride, long long n,
                                          const int* __restrict__ info, int* __restrict__ hist,
                                          int* __restrict__ cell) {
    const float m = __int_as_float(info[0]);
    const float unit = m > 0.f ? 15.99f / m : 0.f;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        Real x[3];
        load_vals<Real, 3>(tgt, stride, i, 0, x);
        unsigned k = 0;
        for (int j = 0; j < 3; ++j) {
            const float q = 16.f + (float)x[j] * unit;   // NaN and infinities: the first or the last cell
            k |= morton_spread((unsigned)fminf(fmaxf(q, 0.f), 31.f)) << j;
        }
        cell[i] = (int)k;
        atomicAdd(hist + k, 1);
    }
}
// hist: counts -> starts, and a copy of them behind (the scatter's cursors); info[0]: the largest count
static __global__ void __launch_bounds__(1024) order_scan_kernel(int* __restrict__ hist, int* __restrict__ info) {
    __shared__ int ws[32], wm[32];
    constexpr int PER = kOrderCells / 1024;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int c[PER], sum = 0, big = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        c[q] = hist[threadIdx.x * PER + q];
        sum += c[q];
        big = max(big, c[q]);
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
        big = max(big, __shfl_xor_sync(0xffffffffu, big, o));
    }
    if (lane == 31) ws[warp] = incl;
    if (lane == 0) wm[warp] = big;
    __syncthreads();
    int at = incl - sum;
    for (int w = 0; w < 32; ++w) {
        if (w < warp) at += ws[w];
        big = max(big, wm[w]);
    }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        hist[threadIdx.x * PER + q] = at;
        hist[kOrderCells + threadIdx.x * PER + q] = at;
        at += c[q];
    }
    if (threadIdx.x == 0) info[0] = big;
}
static __global__ void order_scatter_kernel(const int* __restrict__ cell, long long n, int* __restrict__ cursor,
                                            int* __restrict__ tmp) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        tmp[atomicAdd(cursor + cell[i], 1)] = (int)i;
}
static __global__ void order_rank_kernel(const int* __restrict__ tmp, const int* __restrict__ cell,
                                         const int* __restrict__ start, const int* __restrict__ info, long long n,
                                         long long n_pad, int* __restrict__ perm) {
    const bool crowd = info[0] > kOrderCrowd;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n_pad;
         q += (long long)gridDim.x * blockDim.x) {
        if (crowd || q >= n) {
            perm[q] = (int)q;
            continue;
        }
        const int i = tmp[q], c = cell[i];
        const int b = start[c], e = c + 1 < kOrderCells ? start[c + 1] : (int)n;
        int rank = 0;
        for (int j = b; j < e; ++j) rank += tmp[j] < i;
        perm[b + rank] = i;
    }
}

inline int grid_for(long long work, int block = 256, int max_blocks = 148 * 16) {
    long long b = (work + block - 1) / block;
    if (b < 1) b = 1;
    if (b > max_blocks) b = max_blocks;
    return (int)b;
}

}  // namespace lddmm
