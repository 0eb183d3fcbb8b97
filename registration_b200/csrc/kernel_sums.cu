// C ABI for the kernel sums kff.applyk / kff.applykdifft
// (py-lddmm/kernelFunctions.f90:1-54, 56-114).
#include <type_traits>

#include "host.h"
#include "internal.h"
#include "ops2.cuh"
#include "pack.cuh"
#include "sweep_dispatch.cuh"

namespace lddmm {

// FP64 sums may add their sources in any order, so large ones order both point
// sets by cells (launch_order_rows): folds and groups are then compact wherever the
// points come from.  From 2^30 pairs on (1.6 ms; the twelve launches take 35 us), where
// the sources are so many that folds are bounded at all.
// B200, 65,536 x 65,536 points uniform in the unit cube, sigma 0.05: 6.55 -> 4.37 ms.
// Ordered / as they lie, 524,288 x 2,048 points: 2.02 / 1.69 ms at sigma 1, 1.87 / 1.69 at 0.05.
struct Ordered64 {
    OrderRows t, s;
    float4* src = nullptr;
    bool taken = false;
};
template <class Op>
Ordered64 take_ordered64(Workspace& ws, const SinglePlan& pl, long long n, long long m) {
    Ordered64 o;
    if (sizeof(typename Op::Real) != 8 || pl.n_folds <= kBoundFolds || n < 2048 || n < (1LL << 30) / m) return o;
    o.taken = true;
    o.t = take_order(ws, pl.n_tpad);
    o.s = take_order(ws, pl.m_pad);
    o.src = ws.take<float4>((size_t)Op::NS * pl.m_pad);
    return o;
}
inline int launch_ordered64(const Ordered64& o, const float4* tgt, const float4* src, const SinglePlan& pl,
                            long long n, long long m, int V, float4* boxes, cudaStream_t st) {
    LDDMM_TRY(launch_order_rows<double>(o.t, tgt, n, pl.n_tpad, st));
    LDDMM_TRY(launch_order_rows<double>(o.s, src, m, pl.m_pad, st));
    permute_records_kernel<<<grid_for(pl.m_pad), 256, 0, st>>>(src, o.s.perm, pl.m_pad, m, V, o.src, boxes);
    return cuda_check(cudaGetLastError(), "ordered sum");
}

// ---------------------------------------------------------------------------
// applyk
// ---------------------------------------------------------------------------
struct ApplyKArgs {
    const double* x;
    long long n;
    const double* y;
    long long m;
    const double* beta;
    int d, dimb;
    double sigma;
    int order;
    double* f;
    int split_cap;  // 0: no cap on the number of source chunks
};

template <class Real, int KIND, int DEG, int D, int DIMB>
int applyk_group(const ApplyKArgs& a, int col0, Workspace& ws, cudaStream_t st) {
    // FP32: packed-pair operator (two targets per slot, list source records);
    // FP64: the plain operator on double records.
    using Op = std::conditional_t<sizeof(Real) == 4, OpApplyK2<KIND, DEG, D, DIMB>, OpApplyK<Real, KIND, DEG, D, DIMB>>;
    const SinglePlan pl = plan_single<Op>(a.n, a.m, a.split_cap);
    float4* tgt = ws.take<float4>((size_t)Op::PP * pl.n_tpad);
    float4* src = ws.take<float4>((size_t)Op::NS * pl.m_pad);
    float4* boxes = pl.take_boxes<Op>(ws);
    double* part = ws.take<double>(pl.part_doubles(DIMB));
    int* counters = ws.take<int>(pl.split > 1 ? pl.counters() : 0);
    // sums over the targets' own points (the query cannot know: room for the order whenever n == m)
    const Ordered64 both = take_ordered64<Op>(ws, pl, a.n, a.m);
    OrderRows order = !both.taken && a.n == a.m ? take_order_rows(ws, pl) : OrderRows{};
    double* center = ws.take<double>(kCenterWords);
    if (ws.measuring()) return LDDMM_OK;
    if (ws.overflow()) {
        set_error("workspace too small: need %zu bytes, got %zu", ws.off, ws.cap);
        return LDDMM_ERR_WORKSPACE;
    }
    const KScale ks = kernel_scale(KIND, a.order, a.sigma, !pl.seq);
    typename Op::Params P{};
    P.src4 = src;
    P.src_stride = pl.m_pad;
    P.tgt4 = tgt;
    P.tgt_stride = pl.n_tpad;
    set_poly(P, ks);
    Gather g{};
    g.src = a.beta;
    g.row_stride = a.dimb;
    g.nvals = std::min(DIMB, a.dimb - col0);
    for (int c = 0; c < g.nvals; ++c) g.off[c] = col0 + c;
    g.mult = 1.0;
    launch_bbox_center(a.x, a.n, a.y, a.m, a.d, center, st);
    pack_sum_kernel<Real, sizeof(Real) == 4><<<grid_for(pl.n_tpad + pl.m_pad), 256, 0, st>>>(
        a.x, a.n, Gather{}, 0, tgt, pl.n_tpad, a.y, a.m, g, D, DIMB, src, pl.m_pad, a.d, ks.scale, center, boxes,
        counters, pl.split > 1 ? (int)pl.counters() : 0);
    if (a.x != a.y) order.perm = nullptr;
    LDDMM_TRY((launch_order_rows<Real>(order, tgt, a.n, pl.n_tpad, st)));
    if (both.taken) {
        LDDMM_TRY(launch_ordered64(both, tgt, src, pl, a.n, a.m, DIMB, boxes, st));
        P.src4 = both.src;
        order = both.t;
    }
    // the epilogue writes only the group's own columns
    const EpiSum E{a.f, a.dimb, col0, g.nvals, 1.0};
    return launch_single<Op, false>(pl, a.n, P, boxes, part, st, 0, counters, E, order.perm, a.x == a.y && !both.taken);
}

template <class Real>
int applyk_run(const ApplyKArgs& a, Workspace& ws, cudaStream_t st) {
    // column groups of at most 4 weights; workspace is reused group after group
    const size_t off0 = ws.off;
    size_t peak = off0;
    for (int col0 = 0; col0 < a.dimb; col0 += 4) {
        ws.off = off0;
        const int g = std::min(4, a.dimb - col0);
        int rc = dispatch_kind_p(a.order, [&](auto kind, auto deg) {
            return dispatch_d(a.d, [&](auto D) {
                return dispatch_dimb(g, [&](auto B) {
                    return applyk_group<Real, decltype(kind)::value, decltype(deg)::value, decltype(D)::value,
                                        decltype(B)::value>(a, col0, ws, st);
                });
            });
        });
        if (rc != LDDMM_OK) return rc;
        peak = std::max(peak, ws.off);
    }
    ws.off = peak;
    return LDDMM_OK;
}

static int applyk_validate(const ApplyKArgs& a) {
    if (a.n < 0 || a.m < 0 || a.d < 1 || a.d > 3 || a.dimb < 1 || !(a.sigma > 0) || a.order < 0) {
        set_error("applyk: invalid arguments (n=%lld m=%lld d=%d dimb=%d sigma=%g order=%d); d must be 1..3",
                  a.n, a.m, a.d, a.dimb, a.sigma, a.order);
        return LDDMM_ERR_ARG;
    }
    if (a.n > (1LL << 30) || a.m > (1LL << 30)) {
        set_error("applyk: more than 2^30 points");
        return LDDMM_ERR_ARG;
    }
    if (a.n == 0) return LDDMM_OK;
    LDDMM_TRY(check_device_ptr(a.x, "x"));
    LDDMM_TRY(check_device_ptr(a.f, "f"));
    if (a.m > 0) {
        LDDMM_TRY(check_device_ptr(a.y, "y"));
        LDDMM_TRY(check_device_ptr(a.beta, "beta"));
    }
    return LDDMM_OK;
}

template <class Real>
size_t applyk_ws(int64_t n, int64_t m, int d, int dimb) {
    ApplyKArgs a{nullptr, n, nullptr, m, nullptr, d, dimb, 1.0, 10, nullptr, 0};
    if (n <= 0 || m <= 0 || d < 1 || d > 3 || dimb < 1) return 0;
    Workspace ws;
    applyk_run<Real>(a, ws, 0);
    return ws.off + 256;
}

template <class Real>
int applyk_entry(const ApplyKArgs& a, void* wsp, size_t wsb, cudaStream_t st) {
    LDDMM_TRY(applyk_validate(a));
    if (a.n == 0) return LDDMM_OK;
    if (a.m == 0)
        return cuda_check(cudaMemsetAsync(a.f, 0, sizeof(double) * a.n * a.dimb, st), "applyk memset");
    if (wsp == nullptr) {
        set_error("applyk: workspace is NULL (query the *_workspace function)");
        return LDDMM_ERR_WORKSPACE;
    }
    LDDMM_TRY(check_device_ptr(wsp, "workspace"));
    Workspace ws;
    ws.base = static_cast<char*>(wsp);
    ws.cap = wsb;
    // a first measuring pass so no launch happens with a short workspace
    Workspace meas;
    applyk_run<Real>(a, meas, st);
    if (meas.off > wsb) {
        set_error("applyk: workspace too small: need %zu bytes, got %zu", meas.off, wsb);
        return LDDMM_ERR_WORKSPACE;
    }
    return applyk_run<Real>(a, ws, st);
}

// ---------------------------------------------------------------------------
// applykdifft
// ---------------------------------------------------------------------------
struct DiffKTArgs {
    const double* x;
    long long n;
    const double* y;
    long long m;
    const double* a1;
    const double* a2;
    int na, d, dimb;
    double sigma;
    int order;
    double* f;
};

template <class Real, int KIND, int DEG, int D, int W>
int difft_impl(const DiffKTArgs& a, Workspace& ws, cudaStream_t st) {
    using Op = std::conditional_t<sizeof(Real) == 4, OpDiffKT2<KIND, DEG, D, W>, OpDiffKT<Real, KIND, DEG, D, W>>;
    constexpr int NT = (sizeof(Real) == 4) ? 1 + (W + 3) / 4 : Op::NS;  // target planes
    const SinglePlan pl = plan_single<Op>(a.n, a.m);
    float4* tgt = ws.take<float4>((size_t)NT * pl.n_tpad);
    float4* src = ws.take<float4>((size_t)Op::NS * pl.m_pad);
    float4* boxes = pl.take_boxes<Op>(ws);
    double* part = ws.take<double>(pl.part_doubles(D));
    int* counters = ws.take<int>(pl.counters());
    const Ordered64 both = take_ordered64<Op>(ws, pl, a.n, a.m);
    OrderRows order = !both.taken && a.n == a.m ? take_order_rows(ws, pl) : OrderRows{};
    double* center = ws.take<double>(kCenterWords);
    if (ws.measuring()) return LDDMM_OK;
    const KScale ks = kernel_scale(KIND, a.order, a.sigma, !pl.seq);
    typename Op::Params P{};
    P.src4 = src;
    P.src_stride = pl.m_pad;
    P.tgt4 = tgt;
    P.tgt_stride = pl.n_tpad;
    set_poly(P, ks);
    // u_k / v_l: value w = c*na + i  <->  a[i, row, c]  (the Fortran sum order)
    Gather gu{}, gv{};
    gu.src = a.a1;
    gv.src = a.a2;
    gu.row_stride = gv.row_stride = a.dimb;
    gu.nvals = gv.nvals = a.na * a.dimb;
    gu.mult = gv.mult = 1.0;
    for (int w = 0; w < a.na * a.dimb; ++w) {
        const int i = w % a.na, c = w / a.na;
        gu.off[w] = (long long)i * a.n * a.dimb + c;
        gv.off[w] = (long long)i * a.m * a.dimb + c;
    }
    launch_bbox_center(a.x, a.n, a.y, a.m, a.d, center, st);
    pack_sum_kernel<Real, sizeof(Real) == 4><<<grid_for(pl.n_tpad + pl.m_pad), 256, 0, st>>>(
        a.x, a.n, gu, W, tgt, pl.n_tpad, a.y, a.m, gv, D, W, src, pl.m_pad, a.d, ks.scale, center, boxes, counters,
        (int)pl.counters());
    if (a.x != a.y) order.perm = nullptr;
    LDDMM_TRY((launch_order_rows<Real>(order, tgt, a.n, pl.n_tpad, st)));
    if (both.taken) {
        LDDMM_TRY(launch_ordered64(both, tgt, src, pl, a.n, a.m, W, boxes, st));
        P.src4 = both.src;
        order = both.t;
    }
    const EpiSum E{a.f, a.d, 0, a.d, ks.dscale};   // D may exceed d (d == 1 runs as D == 2)
    return launch_single<Op, false>(pl, a.n, P, boxes, part, st, 0, counters, E, order.perm, a.x == a.y && !both.taken);
}

template <class Real>
int difft_run(const DiffKTArgs& a, Workspace& ws, cudaStream_t st) {
    return dispatch_kind_q(a.order, [&](auto kind, auto deg) {
        return dispatch_d(a.d, [&](auto D) {
            return dispatch_w(a.na * a.dimb, [&](auto W) {
                return difft_impl<Real, decltype(kind)::value, decltype(deg)::value, decltype(D)::value,
                                  decltype(W)::value>(a, ws, st);
            });
        });
    });
}

static int difft_validate(const DiffKTArgs& a) {
    if (a.n < 0 || a.m < 0 || a.d < 1 || a.d > 3 || a.dimb < 1 || a.na < 1 || !(a.sigma > 0) || a.order < 0) {
        set_error("applykdifft: invalid arguments (n=%lld m=%lld na=%d d=%d dimb=%d sigma=%g order=%d)", a.n, a.m,
                  a.na, a.d, a.dimb, a.sigma, a.order);
        return LDDMM_ERR_ARG;
    }
    if (a.order == 0) {
        set_error("applykdifft: the order-0 Laplacian kernel is not differentiable");
        return LDDMM_ERR_ARG;
    }
    if (a.na * a.dimb > 12) {
        set_error("applykdifft: na*dimb = %d exceeds 12", a.na * a.dimb);
        return LDDMM_ERR_UNSUPPORTED;
    }
    if (a.n > (1LL << 30) || a.m > (1LL << 30)) {
        set_error("applykdifft: more than 2^30 points");
        return LDDMM_ERR_ARG;
    }
    if (a.n == 0) return LDDMM_OK;
    LDDMM_TRY(check_device_ptr(a.x, "x"));
    LDDMM_TRY(check_device_ptr(a.a1, "a1"));
    LDDMM_TRY(check_device_ptr(a.f, "f"));
    if (a.m > 0) {
        LDDMM_TRY(check_device_ptr(a.y, "y"));
        LDDMM_TRY(check_device_ptr(a.a2, "a2"));
    }
    return LDDMM_OK;
}

template <class Real>
size_t difft_ws(int64_t n, int64_t m, int na, int d, int dimb) {
    if (n <= 0 || m <= 0 || d < 1 || d > 3 || dimb < 1 || na < 1 || na * dimb > 12) return 0;
    DiffKTArgs a{nullptr, n, nullptr, m, nullptr, nullptr, na, d, dimb, 1.0, 10, nullptr};
    Workspace ws;
    difft_run<Real>(a, ws, 0);
    return ws.off + 256;
}

template <class Real>
int difft_entry(const DiffKTArgs& a, void* wsp, size_t wsb, cudaStream_t st) {
    LDDMM_TRY(difft_validate(a));
    if (a.n == 0) return LDDMM_OK;
    if (a.m == 0)
        return cuda_check(cudaMemsetAsync(a.f, 0, sizeof(double) * a.n * a.d, st), "applykdifft memset");
    Workspace meas;
    difft_run<Real>(a, meas, st);
    if (wsp == nullptr || meas.off > wsb) {
        set_error("applykdifft: workspace too small: need %zu bytes, got %zu", meas.off, wsb);
        return LDDMM_ERR_WORKSPACE;
    }
    LDDMM_TRY(check_device_ptr(wsp, "workspace"));
    Workspace ws;
    ws.base = static_cast<char*>(wsp);
    ws.cap = wsb;
    return difft_run<Real>(a, ws, st);
}

// ---------------------------------------------------------------------------
// applyDivergence
// ---------------------------------------------------------------------------
template <class Real, int KIND, int DEG, int D>
int div_impl(const ApplyKArgs& a, Workspace& ws, cudaStream_t st) {
    using Op = OpDivergence<Real, KIND, DEG, D>;
    const SinglePlan pl = plan_single<Op>(a.n, a.m);
    float4* tgt = ws.take<float4>((size_t)Op::PP * pl.n_tpad);
    float4* src = ws.take<float4>((size_t)Op::NS * pl.m_pad);
    double* part = ws.take<double>(pl.part_doubles(1));
    int* counters = ws.take<int>(pl.counters());
    double* center = ws.take<double>(kCenterWords);
    if (ws.measuring()) return LDDMM_OK;
    const KScale ks = kernel_scale(KIND, a.order, a.sigma, !pl.seq, /*exact_tables=*/true);
    // (the reference's applyDivergence runs on its dense numpy matrices, which
    //  use the exact rational polynomials, kernelFunctions.py:75-88)
    typename Op::Params P{};
    P.src4 = src;
    P.src_stride = pl.m_pad;
    P.tgt4 = tgt;
    P.tgt_stride = pl.n_tpad;
    set_poly(P, ks);
    Gather g{};
    g.src = a.beta;
    g.row_stride = a.d;
    g.nvals = a.d;
    for (int c = 0; c < a.d; ++c) g.off[c] = c;
    g.mult = 1.0;  // K' 2 <x-y, a> = dscale * F * <x'-y', a>
    launch_bbox_center(a.x, a.n, a.y, a.m, a.d, center, st);
    pack_sum_kernel<Real, false><<<grid_for(pl.n_tpad + pl.m_pad), 256, 0, st>>>(
        a.x, a.n, Gather{}, 0, tgt, pl.n_tpad, a.y, a.m, g, D, D, src, pl.m_pad, a.d, ks.scale, center, nullptr,
        counters, (int)pl.counters());
    const EpiSum E{a.f, 1, 0, 1, ks.dscale};
    return launch_single<Op, false>(pl, a.n, P, nullptr, part, st, 0, counters, E);
}

template <class Real>
int div_run(const ApplyKArgs& a, Workspace& ws, cudaStream_t st) {
    return dispatch_kind_q(a.order, [&](auto kind, auto deg) {
        return dispatch_d(a.d, [&](auto D) {
            return div_impl<Real, decltype(kind)::value, decltype(deg)::value, decltype(D)::value>(a, ws, st);
        });
    });
}

template <class Real>
size_t div_ws(int64_t n, int64_t m, int d) {
    if (n <= 0 || m <= 0 || d < 1 || d > 3) return 0;
    ApplyKArgs a{nullptr, n, nullptr, m, nullptr, d, d, 1.0, 10, nullptr, 0};
    Workspace ws;
    div_run<Real>(a, ws, 0);
    return ws.off + 256;
}

template <class Real>
int div_entry(const ApplyKArgs& a, void* wsp, size_t wsb, cudaStream_t st) {
    LDDMM_TRY(applyk_validate(a));
    if (a.order == 0) {
        set_error("applydiv: the order-0 Laplacian kernel is not differentiable");
        return LDDMM_ERR_ARG;
    }
    if (a.n == 0) return LDDMM_OK;
    if (a.m == 0) return cuda_check(cudaMemsetAsync(a.f, 0, sizeof(double) * a.n, st), "applydiv memset");
    Workspace meas;
    div_run<Real>(a, meas, st);
    if (wsp == nullptr || meas.off > wsb) {
        set_error("applydiv: workspace too small: need %zu bytes, got %zu", meas.off, wsb);
        return LDDMM_ERR_WORKSPACE;
    }
    LDDMM_TRY(check_device_ptr(wsp, "workspace"));
    Workspace ws;
    ws.base = static_cast<char*>(wsp);
    ws.cap = wsb;
    return div_run<Real>(a, ws, st);
}

size_t applyk_f32c_scratch_bytes(int64_t n, int64_t m, int d, int dimb, int split_cap) {
    if (n <= 0 || m <= 0 || d < 1 || d > 3 || dimb < 1) return 0;
    ApplyKArgs a{nullptr, n, nullptr, m, nullptr, d, dimb, 1.0, 10, nullptr, split_cap};
    size_t best = 0;
    for (int order : {10, 3}) {  // Gaussian and Laplacian plans
        a.order = order;
        Workspace ws;
        applyk_run<float>(a, ws, 0);
        best = std::max(best, ws.off);
    }
    return best + 256;
}

int applyk_f32c_in_workspace(const double* x, int64_t n, const double* y, int64_t m, const double* beta, int d,
                             int dimb, double sigma, int order, double* f, void* workspace, size_t workspace_bytes,
                             cudaStream_t stream, int split_cap) {
    ApplyKArgs a{x, n, y, m, beta, d, dimb, sigma, order, f, split_cap};
    return applyk_entry<float>(a, workspace, workspace_bytes, stream);
}

}  // namespace lddmm

using namespace lddmm;

extern "C" {

size_t lddmm_applyk_f32c_workspace(int64_t n, int64_t m, int d, int dimb) { return applyk_ws<float>(n, m, d, dimb); }
size_t lddmm_applyk_f64_workspace(int64_t n, int64_t m, int d, int dimb) { return applyk_ws<double>(n, m, d, dimb); }

int lddmm_applyk_f32c(const double* x, int64_t n, const double* y, int64_t m, const double* beta, int d, int dimb,
                      double sigma, int order, double* f, void* workspace, size_t workspace_bytes,
                      lddmm_stream_t stream) {
    ApplyKArgs a{x, n, y, m, beta, d, dimb, sigma, order, f, 0};
    return applyk_entry<float>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

int lddmm_applyk_f64(const double* x, int64_t n, const double* y, int64_t m, const double* beta, int d, int dimb,
                     double sigma, int order, double* f, void* workspace, size_t workspace_bytes,
                     lddmm_stream_t stream) {
    ApplyKArgs a{x, n, y, m, beta, d, dimb, sigma, order, f, 0};
    return applyk_entry<double>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

size_t lddmm_applykdifft_f32c_workspace(int64_t n, int64_t m, int na, int d, int dimb) {
    return difft_ws<float>(n, m, na, d, dimb);
}
size_t lddmm_applykdifft_f64_workspace(int64_t n, int64_t m, int na, int d, int dimb) {
    return difft_ws<double>(n, m, na, d, dimb);
}

int lddmm_applykdifft_f32c(const double* x, int64_t n, const double* y, int64_t m, const double* a1,
                           const double* a2, int na, int d, int dimb, double sigma, int order, double* f,
                           void* workspace, size_t workspace_bytes, lddmm_stream_t stream) {
    DiffKTArgs a{x, n, y, m, a1, a2, na, d, dimb, sigma, order, f};
    return difft_entry<float>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

int lddmm_applykdifft_f64(const double* x, int64_t n, const double* y, int64_t m, const double* a1,
                          const double* a2, int na, int d, int dimb, double sigma, int order, double* f,
                          void* workspace, size_t workspace_bytes, lddmm_stream_t stream) {
    DiffKTArgs a{x, n, y, m, a1, a2, na, d, dimb, sigma, order, f};
    return difft_entry<double>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

size_t lddmm_applydiv_f32c_workspace(int64_t n, int64_t m, int d) { return div_ws<float>(n, m, d); }
size_t lddmm_applydiv_f64_workspace(int64_t n, int64_t m, int d) { return div_ws<double>(n, m, d); }

int lddmm_applydiv_f32c(const double* x, int64_t n, const double* y, int64_t m, const double* a, int d, double sigma,
                        int order, double* f, void* workspace, size_t workspace_bytes, lddmm_stream_t stream) {
    ApplyKArgs q{x, n, y, m, a, d, d, sigma, order, f, 0};
    return div_entry<float>(q, workspace, workspace_bytes, (cudaStream_t)stream);
}

int lddmm_applydiv_f64(const double* x, int64_t n, const double* y, int64_t m, const double* a, int d, double sigma,
                       int order, double* f, void* workspace, size_t workspace_bytes, lddmm_stream_t stream) {
    ApplyKArgs q{x, n, y, m, a, d, d, sigma, order, f, 0};
    return div_entry<double>(q, workspace, workspace_bytes, (cudaStream_t)stream);
}

}  // extern "C"
