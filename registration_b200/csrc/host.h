// Host-side helpers shared by the C-ABI translation units.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <string>

#include "../../include/lddmm_b200.h"
#include "common.cuh"

namespace lddmm {

void set_error(const char* fmt, ...);

// Bump allocator over the caller's workspace.  With base == nullptr it only
// measures, so the *_workspace queries run exactly the same code as the calls.
struct Workspace {
    char* base = nullptr;
    size_t cap = 0;
    size_t off = 0;
    template <class T>
    T* take(size_t count) {
        off = (off + 255) & ~size_t(255);
        T* p = base ? reinterpret_cast<T*>(base + off) : nullptr;
        off += count * sizeof(T);
        return p;
    }
    bool measuring() const { return base == nullptr; }
    bool overflow() const { return base && off > cap; }
};

struct DeviceInfo {
    int device = 0;
    int sms = 148;
};
DeviceInfo device_info();

// Maximum resident blocks per SM of a kernel (cached by the caller per kernel).
int occupancy_blocks(const void* kernel, int block, size_t dyn_smem = 0);

// Number of source chunks of a sweep over n_tb target groups and n_folds folds
// of 32 sources; `resident` blocks fit the device at once, a block's four warps
// share the folds of its chunk.  A function of the operator, the shape and the
// SM count only (workspace queries run the same code).
//   Many blocks (four waves and more): up to 64 blocks per SM, at least 32 folds
// per warp, so that groups whose far folds are passed over balance out.  (With 16 every
// group measures its bounds twice as often: FP64 varifold value of 20,480 cells 576 ->
// 555 us, FP32c current gradient of 30,000 edges, nothing far, 971 -> 940 us.)
//   Fewer: waves count.  The chunks that make ceil(blocks / resident) (folds per
// warp + kBlockFolds) smallest, kBlockFolds being what a block's start and end
// cost in folds (3,166 points, 11 / 8 / 5 chunks: 404 / 392 / 420 us per shot and
// adjoint; 10,242 points, adjoint sweeps with 444 resident blocks: 5 chunks = 405
// blocks 1421 us, 6 chunks = 486 blocks 1542 us).
//   A segment of a ragged launch (`shared`) has the other segments beside it: 8
// folds per warp (template step of 8 x 2,562 points with 4 / 8 / 16: 2792 / 2778 /
// 2945 us, with a lone problem's chunks 3231).
// Varifold gradient of 20,480 cells, 4 / 8 / 16 folds per warp: 431 / 422 / 382 us.
constexpr int kBlockFolds = 3;
inline int choose_split(int n_tb, int n_folds, int sms, int resident, bool shared) {
    if (n_tb <= 0 || n_folds <= 0) return 1;
    const long long want = (64LL * sms + n_tb - 1) / n_tb;
    const long long many = std::max(1LL, std::min<long long>(want, n_folds / (4 * (shared ? 8 : 32))));
    if (shared || many * n_tb >= 4LL * resident) return (int)many;
    // for each number of waves the most chunks that fit, then the fewest with as few folds per warp
    const long long cap = (n_folds + 3) / 4;
    long long best = 1, best_cost = -1;
    for (long long waves = 1; waves <= 5; ++waves) {
        const long long fit = std::min(cap, waves * resident / n_tb);
        if (fit < 1) continue;
        const long long folds = (n_folds + 4 * fit - 1) / (4 * fit);
        const long long cost = waves * (folds + kBlockFolds);
        if (best_cost < 0 || cost < best_cost) {
            best = (n_folds + 4 * folds - 1) / (4 * folds);
            best_cost = cost;
        }
    }
    return (int)best;
}

inline long long round_up(long long v, long long m) { return (v + m - 1) / m * m; }

// Returns LDDMM_ERR_ARG unless ptr is device (or managed) memory.
int check_device_ptr(const void* ptr, const char* name);

inline int cuda_check(cudaError_t e, const char* what) {
    if (e != cudaSuccess) {
        set_error("%s: %s", what, cudaGetErrorString(e));
        return LDDMM_ERR_CUDA;
    }
    return LDDMM_OK;
}

#define LDDMM_TRY(expr)                   \
    do {                                  \
        int _rc = (expr);                 \
        if (_rc != LDDMM_OK) return _rc;  \
    } while (0)

// Laplacian polynomial tables of py-lddmm/kernelFunctions.f90 (c_ :24-26,
// c1_ :85-86, c2_ :325) with their default-real (float32) literal values, or
// (exact = true) the exact rationals of the dense numpy path lapPol /
// lapPolDiff / lapPolDiff2 (kernelFunctions.py:58-103).
void laplacian_tables(int order, double P[5], double Q[4], double Rr[3], bool exact = false);

}  // namespace lddmm
