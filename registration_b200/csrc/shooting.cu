// Geodesic shooting and its Hamiltonian adjoint, fused per time step.
//
//   lddmm_shoot_*    : landmarkDirectEvolutionEuler (py-lddmm/pointEvolution.py:666-730)
//                      x_{t+1} = x_t + dt K(x_t, x_t) a_t, dt = 1/T, plus the
//                      regularisation energy sum_t rw dt <a_t, K(x_t) a_t> of
//                      objectiveFunDef (surfaceMatching.py:205-212), computed
//                      from the same kernel sums.
//   lddmm_covector_* : landmarkHamiltonianCovector / Gradient (pointEvolution.py:735-817)
//                      p_t = p_{t+1} + dt applyDiffKT(x_t, [p, a, -2 rw a], [a, p, a]),
//                      dat_t = 2 rw a_t - p_{t+1}.
//   lddmm_epdiff_*   : landmarkEPDiff (pointEvolution.py:599-658).
//
// The 3-momentum inner product of the adjoint is rewritten as
//   <p_k,a_l> + <a_k,p_l> - 2 rw <a_k,a_l> = <p_k - 2 rw a_k, a_l> + <a_k, p_l>,
// a 2d-wide dot (u_k = (p_k - 2 rw a_k, a_k), v_l = (a_l, p_l)).
//
// One time step of a shot or adjoint = one sweep over (target group, source chunk)
// items, whose epilogue adds a group's chunks in a fixed order, applies the Euler
// (or adjoint) update in FP64 and writes the packed planes of the next step and the
// step's energy partials (one per group, so the reduction order is fixed).  EPDiff
// keeps a combine kernel per step.
#include "dataterm_fused.cuh"
#include "fused_small.cuh"
#include "host.h"
#include "ops2.cuh"
#include "pack.cuh"
#include "sweep_dispatch.cuh"

namespace lddmm {

constexpr int kCombineThreads = 256;
constexpr int kMaxBatch = 1 << 12;   // trial step sizes per batched call

inline int combine_blocks(long long n) { return (int)std::min<long long>(1024, (n + kCombineThreads - 1) / kCombineThreads); }

// the packing frame: (v - c) * s, c the bounding-box centre of the initial points
template <class Real>
LDDMM_D void store_point(float4* planes, long long stride, long long i, const double* v, int d, double s,
                         const double* c) {
    double q[4] = {0, 0, 0, 0};
    for (int j = 0; j < d; ++j) q[j] = (v[j] - c[j]) * s;
    if constexpr (sizeof(Real) == 4) {
        planes[i] = make_float4((float)q[0], (float)q[1], (float)q[2], 0.f);
    } else {
        double2* o = reinterpret_cast<double2*>(planes);
        o[i] = make_double2(q[0], q[1]);
        o[stride + i] = make_double2(q[2], 0.0);
    }
}

// values v[0..nv) into planes first_plane.. of record i
template <class Real>
LDDMM_D void store_vals(float4* planes, long long stride, long long i, int first_plane, const double* v, int nv,
                        int nslots) {
    constexpr int PW = Traits<Real>::PER_WORD;
    for (int w = 0; w < (nslots + PW - 1) / PW; ++w) {
        Real q[PW];
        for (int j = 0; j < PW; ++j) q[j] = (w * PW + j < nv) ? (Real)v[w * PW + j] : (Real)0;
        float4* dst = planes + (long long)(first_plane + w) * stride + i;
        if constexpr (sizeof(Real) == 4) *dst = make_float4(q[0], q[1], q[2], q[3]);
        else *reinterpret_cast<double2*>(dst) = make_double2(q[0], q[1]);
    }
}

template <class Real>
LDDMM_D void zero_record(float4* planes, long long stride, long long i, int nplanes) {
    for (int p = 0; p < nplanes; ++p) planes[(long long)p * stride + i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// List source record (packed-pair FP32 operators, ops2.cuh): values
// [(x - c) * s for D coordinates, vals[0..nv) padded to V].
LDDMM_D void store_list(float4* planes, long long stride, long long i, const double* x, int d, int D, double s,
                        const double* c, const double* vals, int nv, int V) {
    float v[16];
    for (int q = 0; q < 16; ++q) v[q] = 0.f;
    for (int j = 0; j < d; ++j) v[j] = (float)((x[j] - c[j]) * s);
    for (int q = 0; q < nv && q < V; ++q) v[D + q] = (float)vals[q];
    for (int w = 0; w < (D + V + 3) / 4; ++w)
        planes[(long long)w * stride + i] = make_float4(v[4 * w], v[4 * w + 1], v[4 * w + 2], v[4 * w + 3]);
}

// Fold box of source row i (whole warps, see store_fold_box): packed position of x, the
// values v[0..nv) of its NW columns.
template <class Real, int NW>
LDDMM_D void store_box(float4* boxes, long long i, bool valid, const double* x, const double* v, int nv, int nw, int d,
                       double s, const double* c) {
    if (boxes == nullptr) return;
    Real p[3] = {0, 0, 0}, w[NW];
    if (valid)
        for (int j = 0; j < d; ++j) p[j] = (Real)((x[j] - c[j]) * s);
#pragma unroll
    for (int j = 0; j < NW; ++j) w[j] = valid && j < nv ? (Real)v[j] : (Real)0;
    store_fold_box<Real, NW>(boxes, i, valid, p, w, nw);
}

// ---- shooting ---------------------------------------------------------------
// Packed planes of one step: a sweep reads one set while its epilogue writes the other.
struct StepPlanes {
    float4 *tgt, *src, *boxes;
};

// Packs step-0 planes: targets (pos) and sources (pos, a); pads both sets, copies
// x to xt[0], zeroes the counters.
template <class Real, bool LIST>
static __global__ void shoot_pack_kernel(const double* __restrict__ x, const double* __restrict__ a, long long n,
                                         int d, double s, const double* __restrict__ c, StepPlanes p0, StepPlanes p1,
                                         long long tstride, long long sstride, int pp, int nslots, int ns,
                                         double* __restrict__ xt0, int* __restrict__ counters, int n_counters) {
    const long long npad = tstride > sstride ? tstride : sstride;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npad;
         i += (long long)gridDim.x * blockDim.x) {
        if (i < n_counters) counters[i] = 0;
        if (i < sstride) store_box<Real, 3>(p0.boxes, i, i < n, x + i * d, a + i * d, d, nslots, d, s, c);
        if (i < n) {
            for (int j = 0; j < d; ++j) xt0[i * d + j] = x[i * d + j];
            store_point<Real>(p0.tgt, tstride, i, x + i * d, d, s, c);
            if constexpr (LIST) {
                store_list(p0.src, sstride, i, x + i * d, d, nslots, s, c, a + i * d, d, nslots);
            } else {
                store_point<Real>(p0.src, sstride, i, x + i * d, d, s, c);
                store_vals<Real>(p0.src, sstride, i, pp, a + i * d, d, nslots);
            }
        } else {
            if (i < tstride) {
                zero_record<Real>(p0.tgt, tstride, i, pp);
                zero_record<Real>(p1.tgt, tstride, i, pp);
            }
            if (i < sstride) {
                zero_record<Real>(p0.src, sstride, i, ns);
                zero_record<Real>(p1.src, sstride, i, ns);
            }
        }
    }
}

// v = the group's sums; x1 = x0 + dt v; energy partial <a, v>; pack next step.
// The last step's last group adds the energy.
template <class Real, bool LIST>
struct EpiShoot {
    static constexpr bool NONE = false;
    int d, pp, nslots;
    double dt, s;
    const double* c;
    const double *x0, *a0;
    double* x1;
    const double* a1;   // next step's momenta, NULL for the last step
    StepPlanes nx;
    long long tstride, sstride;
    double* epart;      // this step's partials, one per group
    // last step: energy = escale * (all steps' partials), if energy
    double* energy;
    const double* eall;
    long long ecount;
    double escale;
    int* counter;
    int groups;
    template <int GT, int NOUT>
    LDDMM_D void run(const SegDesc& sg, int tb, const int* srow, const double* red) const {
        double e = 0.0;
        for (int r = threadIdx.x; r < GT; r += blockDim.x) {
            const long long i = srow[r];
            const bool valid = i < sg.n_tgt;
            if (sg.perm == nullptr && srow[r & ~31] >= sg.n_tgt) continue;   // whole warps: fold boxes
            double xn[3] = {0, 0, 0};
            for (int j = 0; j < d && valid; ++j) {
                const double v = red[r * NOUT + j];
                e += a0[i * d + j] * v;
                xn[j] = x0[i * d + j] + dt * v;
                x1[i * d + j] = xn[j];
            }
            if (a1 == nullptr) continue;
            if (sg.perm == nullptr) store_box<Real, 3>(nx.boxes, i, valid, xn, a1 + i * d, d, nslots, d, s, c);
            if (!valid) continue;
            store_point<Real>(nx.tgt, tstride, i, xn, d, s, c);
            if constexpr (LIST) {
                store_list(nx.src, sstride, i, xn, d, nslots, s, c, a1 + i * d, d, nslots);
            } else {
                store_point<Real>(nx.src, sstride, i, xn, d, s, c);
                store_vals<Real>(nx.src, sstride, i, pp, a1 + i * d, d, nslots);
            }
        }
        e = block_sum_all(e);
        if (threadIdx.x == 0) epart[tb] = e;
        if (energy == nullptr || !last_block(counter, groups)) return;
        double t = 0.0;
        for (long long q = threadIdx.x; q < ecount; q += blockDim.x) t += __ldcg(eall + q);
        t = block_sum_all(t);
        if (threadIdx.x == 0) *energy = escale * t;
    }
};

struct ShootArgs {
    const double* x0;
    long long n;
    int d;
    const double* at;
    int T;
    double dt;  // Euler step; <= 0 means 1/T
    double sigma;
    int order;
    double rw;
    double* xt;
    double* energy;
    // optional search direction: the shot's momenta are at - (*eps) dir, written to at_try
    const double* dir = nullptr;
    const double* eps = nullptr;
    double* at_try = nullptr;
    // batched trial steps: nbatch step sizes eps[0..nbatch), outputs at_try, xt, energy stacked per candidate
    int nbatch = 1;
};

// at_try = at - (*eps) dir, rounded as two FP64 operations (the trial step of a line search)
static __global__ void trial_momenta_kernel(const double* __restrict__ at, const double* __restrict__ dir,
                                            const double* __restrict__ eps, long long count,
                                            double* __restrict__ at_try) {
    const double e = *eps;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count;
         i += (long long)gridDim.x * blockDim.x)
        at_try[i] = __dsub_rn(at[i], __dmul_rn(e, dir[i]));
}

template <class Real, int KIND, int DEG, int D, bool SMALL = false>
int shoot_impl(const ShootArgs& a, Workspace& ws, cudaStream_t st) {
    constexpr bool LIST = sizeof(Real) == 4;  // FP32: packed-pair operator with list records
    using Op = std::conditional_t<LIST, OpApplyK2<KIND, DEG, D, D, SMALL>, OpApplyK<Real, KIND, DEG, D, D>>;
    const SinglePlan pl = plan_single<Op>(a.n, a.n);
    StepPlanes pn[2];
    for (StepPlanes& p : pn) {
        p.tgt = ws.take<float4>((size_t)Op::PP * pl.n_tpad);
        p.src = ws.take<float4>((size_t)Op::NS * pl.m_pad);
        p.boxes = pl.take_boxes<Op>(ws, LIST ? kBoundFoldsPacked : kBoundFolds);
    }
    double* part = ws.take<double>(pl.part_doubles(D));
    int* counters = ws.take<int>(pl.counters());
    OrderRows order = take_order_rows(ws, pl);
    double* epart = ws.take<double>((size_t)a.T * pl.n_tb);
    double* center = ws.take<double>(kCenterWords);
    if (ws.measuring()) return LDDMM_OK;
    const KScale ks = kernel_scale(KIND, a.order, a.sigma, !pl.seq);
    typename Op::Params P{};
    P.src_stride = pl.m_pad;
    P.tgt_stride = pl.n_tpad;
    set_poly(P, ks);
    const long long N = a.n * a.d;
    launch_bbox_center(a.x0, a.n, nullptr, 0, a.d, center, st);
    shoot_pack_kernel<Real, LIST><<<grid_for(std::max(pl.n_tpad, pl.m_pad)), 256, 0, st>>>(
        a.x0, a.at, a.n, a.d, ks.scale, center, pn[0], pn[1], pl.n_tpad, pl.m_pad, Op::PP, D, Op::NS, a.xt, counters,
        (int)pl.counters());
    LDDMM_TRY((launch_order_rows<Real>(order, pn[0].tgt, a.n, pl.n_tpad, st)));
    const double dt = a.dt > 0 ? a.dt : 1.0 / a.T;
    for (int t = 0; t < a.T; ++t) {
        const StepPlanes& p = pn[t & 1];
        P.tgt4 = p.tgt;
        P.src4 = p.src;
        const bool last = t + 1 == a.T;
        EpiShoot<Real, LIST> E{a.d, Op::PP, D, dt, ks.scale, center, a.xt + t * N, a.at + t * N, a.xt + (t + 1) * N,
                               last ? nullptr : a.at + (t + 1) * N, pn[(t + 1) & 1], pl.n_tpad, pl.m_pad,
                               epart + (long long)t * pl.n_tb, last ? a.energy : nullptr, epart,
                               (long long)a.T * pl.n_tb, a.rw * dt, counters + pl.n_tb, pl.n_tb};
        LDDMM_TRY((launch_single<Op, false>(pl, a.n, P, p.boxes, part, st, 0, counters, E, order.perm)));
        if (order.perm != nullptr && !last)   // the epilogue's rows are not whole folds
            fold_boxes_kernel<Real, LIST><<<grid_for(pl.m_pad), 256, 0, st>>>(
                pn[(t + 1) & 1].src, pl.m_pad, a.n, D, D, pn[(t + 1) & 1].boxes);
    }
    return LDDMM_OK;
}

// n <= kFusedMaxPoints (and d >= 2): all T steps in one cluster launch (fused_small.cuh)
template <class Real, int KIND, int DEG, int D>
int shoot_fused(const ShootArgs& a, Workspace& ws, cudaStream_t st) {
    const FusedShape fs = fused_shape(a.n);
    double* epart = ws.take<double>((size_t)kFusedMaxCluster * a.nbatch);
    if (ws.measuring()) return LDDMM_OK;
    const KScale ks = kernel_scale(KIND, a.order, a.sigma, sizeof(Real) == 4);
    FusedCoef cf{};
    for (int j = 0; j < 5; ++j) cf.pk[j] = ks.pk[j];
    for (int j = 0; j < 4; ++j) cf.pq[j] = ks.pq[j];
    const double dt = a.dt > 0 ? a.dt : 1.0 / a.T;
    return launch_fused(shoot_fused_kernel<Real, KIND, DEG, D>, fs, a.nbatch, fused_dyn_smem<Real>(a.n, D),
                        fused_dyn_smem<Real>(kFusedMaxPoints, 3), st, a.x0, a.at,
                        (long long)a.n, a.T, dt, ks.scale, cf, a.rw, fs, a.xt, a.energy, epart, a.dir, a.eps,
                        a.at_try);
}

template <class Real>
int shoot_run(const ShootArgs& a0, Workspace& ws, cudaStream_t st) {
    ShootArgs a = a0;
    const bool fused = a.n <= kFusedMaxPoints && a.d >= 2;
    if (a.nbatch > 1 && !fused) {
        // general path: the candidates one after the other, each on the same workspace
        const long long N = a.n * a.d;
        const size_t off0 = ws.off;
        size_t top = off0;
        for (int b = 0; b < a.nbatch; ++b) {
            ShootArgs q = a;
            q.nbatch = 1;
            q.eps = a.eps ? a.eps + b : nullptr;
            q.at_try = a.at_try ? a.at_try + (long long)b * a.T * N : nullptr;
            q.xt = a.xt ? a.xt + (long long)b * (a.T + 1) * N : nullptr;
            q.energy = a.energy ? a.energy + b : nullptr;
            ws.off = off0;
            LDDMM_TRY(shoot_run<Real>(q, ws, st));
            top = std::max(top, ws.off);
        }
        ws.off = top;
        return LDDMM_OK;
    }
    if (a.dir != nullptr && !fused) {
        // general path: form the trial momenta, then shoot them
        if (!ws.measuring()) {
            const long long cnt = (long long)a.T * a.n * a.d;
            trial_momenta_kernel<<<grid_for(cnt), 256, 0, st>>>(a.at, a.dir, a.eps, cnt, a.at_try);
        }
        a.at = a.at_try;
        a.dir = nullptr;
    }
    return dispatch_kind_p(a.order, [&](auto kind, auto deg) {
        return dispatch_d(a.d, [&](auto D) {
            constexpr int K_ = decltype(kind)::value, P_ = decltype(deg)::value, D_ = decltype(D)::value;
            if (a.n <= kFusedMaxPoints && a.d == D_) return shoot_fused<Real, K_, P_, D_>(a, ws, st);
            if (a.n <= kSmallTargets) return shoot_impl<Real, K_, P_, D_, true>(a, ws, st);
            return shoot_impl<Real, K_, P_, D_>(a, ws, st);
        });
    });
}

// ---- covector ---------------------------------------------------------------
// planes of step t: targets (pos, u = (p - 2 rw a, a)), sources (pos, v = (a, p))
template <class Real, bool LIST>
LDDMM_D void cov_store(float4* tgt, long long tstride, float4* src, long long sstride, long long i, int pp,
                       const double* x, const double* a, const double* p, int d, double s, const double* c,
                       double rw, int tw) {
    double u[8], v[8];
    for (int j = 0; j < d; ++j) {
        u[j] = p[j] - 2.0 * rw * a[j];
        u[d + j] = a[j];
        v[j] = a[j];
        v[d + j] = p[j];
    }
    if (i < tstride) {
        store_point<Real>(tgt, tstride, i, x, d, s, c);
        store_vals<Real>(tgt, tstride, i, pp, u, 2 * d, tw);
    }
    if (i < sstride) {
        if constexpr (LIST) {
            store_list(src, sstride, i, x, d, tw / 2, s, c, v, 2 * d, tw);
        } else {
            store_point<Real>(src, sstride, i, x, d, s, c);
            store_vals<Real>(src, sstride, i, pp, v, 2 * d, tw);
        }
    }
}

template <class Real>
LDDMM_D void cov_box(float4* boxes, long long i, bool valid, const double* x, const double* a, const double* p, int d,
                     double s, const double* c, int tw) {
    if (boxes == nullptr) return;
    double v[6] = {0, 0, 0, 0, 0, 0};
    for (int j = 0; j < d && valid; ++j) {
        v[j] = a[j];
        v[d + j] = p[j];
    }
    store_box<Real, 6>(boxes, i, valid, x, v, 2 * d, tw, d, s, c);
}

// Packs the planes of step T-1; pads both sets, copies p to pxt[T], zeroes the counters.
template <class Real, bool LIST>
static __global__ void cov_pack_kernel(const double* __restrict__ x, const double* __restrict__ a,
                                       const double* __restrict__ p, long long n, int d, double s,
                                       const double* __restrict__ c, double rw, StepPlanes p0, StepPlanes p1,
                                       long long tstride, long long sstride, int pp, int tplanes, int nplanes, int tw,
                                       double* __restrict__ pT, int* __restrict__ counters, int n_counters) {
    const long long npad = tstride > sstride ? tstride : sstride;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npad;
         i += (long long)gridDim.x * blockDim.x) {
        if (i < n_counters) counters[i] = 0;
        if (i < sstride) cov_box<Real>(p0.boxes, i, i < n, x + i * d, a + i * d, p + i * d, d, s, c, tw);
        if (i < n) {
            for (int j = 0; j < d; ++j) pT[i * d + j] = p[i * d + j];
            cov_store<Real, LIST>(p0.tgt, tstride, p0.src, sstride, i, pp, x + i * d, a + i * d, p + i * d, d, s, c,
                                  rw, tw);
        } else {
            if (i < tstride) {
                zero_record<Real>(p0.tgt, tstride, i, tplanes);
                zero_record<Real>(p1.tgt, tstride, i, tplanes);
            }
            if (i < sstride) {
                zero_record<Real>(p0.src, sstride, i, nplanes);
                zero_record<Real>(p1.src, sstride, i, nplanes);
            }
        }
    }
}

// p_t = p_{t+1} + dt * dscale * sums; dat_t = 2 rw a_t - p_{t+1}; pack step t-1.
template <class Real, bool LIST>
struct EpiCov {
    static constexpr bool NONE = false;
    int d, pp, tw;
    double dt, dscale, rw, s;
    const double* c;
    const double *p_next, *a_t;
    double *p_t, *dat_t;
    const double *x_prev, *a_prev;   // NULL for step 0
    StepPlanes nx;
    long long tstride, sstride;
    template <int GT, int NOUT>
    LDDMM_D void run(const SegDesc& sg, int, const int* srow, const double* red) const {
        for (int r = threadIdx.x; r < GT; r += blockDim.x) {
            const long long i = srow[r];
            const bool valid = i < sg.n_tgt;
            if (sg.perm == nullptr && srow[r & ~31] >= sg.n_tgt) continue;   // whole warps: fold boxes
            double pn[3] = {0, 0, 0};
            for (int j = 0; j < d && valid; ++j) {
                const double pj = p_next[i * d + j];
                pn[j] = pj + dt * (dscale * red[r * NOUT + j]);
                p_t[i * d + j] = pn[j];
                if (dat_t != nullptr) dat_t[i * d + j] = 2.0 * rw * a_t[i * d + j] - pj;
            }
            if (x_prev == nullptr) continue;
            if (sg.perm == nullptr)
                cov_box<Real>(nx.boxes, i, valid, x_prev + i * d, a_prev + i * d, pn, d, s, c, tw);
            if (valid)
                cov_store<Real, LIST>(nx.tgt, tstride, nx.src, sstride, i, pp, x_prev + i * d, a_prev + i * d, pn, d,
                                      s, c, rw, tw);
        }
    }
};

struct CovArgs {
    const double* xt;
    long long n;
    int d;
    const double* at;
    int T;
    double dt;  // Euler step; <= 0 means 1/T
    const double* px1;
    double sigma;
    int order;
    double rw;
    double* pxt;
    double* dat;
};

template <class Real, int KIND, int DEG, int D, bool SMALL = false>
int cov_impl(const CovArgs& a, Workspace& ws, cudaStream_t st) {
    constexpr int W = 2 * D;
    constexpr bool LIST = sizeof(Real) == 4;  // FP32: packed-pair operator with list records
    using Op = std::conditional_t<LIST, OpDiffKT2<KIND, DEG, D, W, SMALL>, OpDiffKT<Real, KIND, DEG, D, W>>;
    constexpr int NT = LIST ? 1 + (W + 3) / 4 : Op::NS;  // target planes (standard layout)
    const SinglePlan pl = plan_single<Op>(a.n, a.n);
    StepPlanes pn[2];
    for (StepPlanes& p : pn) {
        p.tgt = ws.take<float4>((size_t)NT * pl.n_tpad);
        p.src = ws.take<float4>((size_t)Op::NS * pl.m_pad);
        p.boxes = pl.take_boxes<Op>(ws, LIST ? kBoundFoldsPacked : kBoundFolds);
    }
    double* part = ws.take<double>(pl.part_doubles(D));
    int* counters = ws.take<int>(pl.counters());
    OrderRows order = take_order_rows(ws, pl);
    double* center = ws.take<double>(kCenterWords);
    if (ws.measuring()) return LDDMM_OK;
    const KScale ks = kernel_scale(KIND, a.order, a.sigma, !pl.seq);
    typename Op::Params P{};
    P.src_stride = pl.m_pad;
    P.tgt_stride = pl.n_tpad;
    set_poly(P, ks);
    const long long N = a.n * a.d;
    const double dt = a.dt > 0 ? a.dt : 1.0 / a.T;
    const int T = a.T;
    launch_bbox_center(a.xt, a.n, nullptr, 0, a.d, center, st);
    cov_pack_kernel<Real, LIST><<<grid_for(std::max(pl.n_tpad, pl.m_pad)), 256, 0, st>>>(
        a.xt + (long long)(T - 1) * N, a.at + (long long)(T - 1) * N, a.px1, a.n, a.d, ks.scale, center, a.rw,
        pn[(T - 1) & 1], pn[T & 1], pl.n_tpad, pl.m_pad, Op::PP, NT, Op::NS, W, a.pxt + (long long)T * N, counters,
        (int)pl.counters());
    LDDMM_TRY((launch_order_rows<Real>(order, pn[(T - 1) & 1].tgt, a.n, pl.n_tpad, st)));
    for (int t = T - 1; t >= 0; --t) {
        const StepPlanes& p = pn[t & 1];
        P.tgt4 = p.tgt;
        P.src4 = p.src;
        EpiCov<Real, LIST> E{a.d, Op::PP, W, dt, ks.dscale, a.rw, ks.scale, center, a.pxt + (long long)(t + 1) * N,
                             a.at + (long long)t * N, a.pxt + (long long)t * N,
                             a.dat ? a.dat + (long long)t * N : nullptr,
                             t > 0 ? a.xt + (long long)(t - 1) * N : nullptr,
                             t > 0 ? a.at + (long long)(t - 1) * N : nullptr, pn[(t + 1) & 1], pl.n_tpad, pl.m_pad};
        LDDMM_TRY((launch_single<Op, false>(pl, a.n, P, p.boxes, part, st, 0, counters, E, order.perm)));
        if (order.perm != nullptr && t > 0)   // the epilogue's rows are not whole folds
            fold_boxes_kernel<Real, LIST><<<grid_for(pl.m_pad), 256, 0, st>>>(
                pn[(t + 1) & 1].src, pl.m_pad, a.n, D, W, pn[(t + 1) & 1].boxes);
    }
    return LDDMM_OK;
}

template <class Real, int KIND, int QDEG, int D>
int cov_fused(const CovArgs& a, Workspace& ws, cudaStream_t st) {
    const FusedShape fs = fused_shape(a.n);
    if (ws.measuring()) return LDDMM_OK;
    const KScale ks = kernel_scale(KIND, a.order, a.sigma, sizeof(Real) == 4);
    FusedCoef cf{};
    for (int j = 0; j < 5; ++j) cf.pk[j] = ks.pk[j];
    for (int j = 0; j < 4; ++j) cf.pq[j] = ks.pq[j];
    const double dt = a.dt > 0 ? a.dt : 1.0 / a.T;
    return launch_fused(cov_fused_kernel<Real, KIND, QDEG, D>, fs, 1, fused_dyn_smem<Real>(a.n, D),
                        fused_dyn_smem<Real>(kFusedMaxPoints, 3), st, a.xt, a.at,
                        a.px1, (long long)a.n, a.T, dt, ks.scale, ks.dscale, cf, a.rw, fs, a.pxt, a.dat);
}

template <class Real>
int cov_run(const CovArgs& a, Workspace& ws, cudaStream_t st) {
    return dispatch_kind_q(a.order, [&](auto kind, auto deg) {
        return dispatch_d(a.d, [&](auto D) {
            constexpr int K_ = decltype(kind)::value, Q_ = decltype(deg)::value, D_ = decltype(D)::value;
            if (a.n <= kFusedMaxPoints && a.d == D_) return cov_fused<Real, K_, Q_, D_>(a, ws, st);
            if (a.n <= kSmallTargets) return cov_impl<Real, K_, Q_, D_, true>(a, ws, st);
            return cov_impl<Real, K_, Q_, D_>(a, ws, st);
        });
    });
}

// ---- EPDiff -------------------------------------------------------------------
// x_{k+1} = x_k + dt K a_k ; a_{k+1} = a_k - dt applyDiffKT(x_k, [a_k], [a_k]).
// Two sums over the same pairs, computed by one operator.
template <class Real_, int KIND, int PDEG, int QDEG, int D>
struct OpEPDiff {
    using Real = Real_;
    static constexpr bool F32 = sizeof(Real) == 4;
    static constexpr int FAMILY = KIND;
    static constexpr int TPS = 1;
    static constexpr int R = 2;
    static constexpr int PP = PointPlanes<Real>::N;
    static constexpr int WP = (D + Traits<Real>::PER_WORD - 1) / Traits<Real>::PER_WORD;
    static constexpr int NS = PP + WP;
    static constexpr int NOUT = 2 * D;
    using Params = KernelParamsBase<Real>;
    using Acc = typename AccFor<Real>::template type<2 * D>;
    struct Tgt {
        Real x[D];
        Real a[D];
    };
    struct Src {
        Real y[D];
        Real a[D];
    };
    static LDDMM_D void load_target(const Params& P, long long row, Tgt& t) {
        load_vals<Real, D>(P.tgt4, P.tgt_stride, row, 0, t.x);
        load_vals<Real, D>(P.tgt4, P.tgt_stride, row, PP, t.a);
    }
    static LDDMM_D void load_source(const float4* S, int j, Src& s) {
        load_vals_smem<Real, D>(S, j, 0, s.y);
        load_vals_smem<Real, D>(S, j, PP, s.a);
    }
    template <bool LIB = false>
    static LDDMM_D void pair(const Params& P, const Tgt& t, const Src& s, Acc& acc) {
        Real dx[D], r2 = 0, dot = 0;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            dx[j] = t.x[j] - s.y[j];
            r2 = j == 0 ? dx[j] * dx[j] : r2 + dx[j] * dx[j];
            dot = j == 0 ? t.a[j] * s.a[j] : dot + t.a[j] * s.a[j];
        }
        const Real k = kval<Real, KIND, PDEG, LIB>(P.pk, r2);
        const Real g = kdiff<Real, KIND, QDEG, LIB>(P.pq, r2) * dot;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            acc.fma(j, k, s.a[j]);
            acc.fma(D + j, g, dx[j]);
        }
    }
};

template <class Real>
static __global__ void epd_pack_kernel(const double* __restrict__ x, const double* __restrict__ a, long long n,
                                       int d, double s, const double* __restrict__ c, float4* tgt, long long tstride,
                                       float4* src, long long sstride, int pp, int nslots, int ns) {
    const long long npad = tstride > sstride ? tstride : sstride;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npad;
         i += (long long)gridDim.x * blockDim.x) {
        if (i < n) {
            if (i < tstride) {
                store_point<Real>(tgt, tstride, i, x + i * d, d, s, c);
                store_vals<Real>(tgt, tstride, i, pp, a + i * d, d, nslots);
            }
            if (i < sstride) {
                store_point<Real>(src, sstride, i, x + i * d, d, s, c);
                store_vals<Real>(src, sstride, i, pp, a + i * d, d, nslots);
            }
        } else {
            if (i < tstride) zero_record<Real>(tgt, tstride, i, ns);
            if (i < sstride) zero_record<Real>(src, sstride, i, ns);
        }
    }
}

template <class Real>
static __global__ void epd_combine_kernel(const double* __restrict__ part, long long n, int d, int dout, int split,
                                          double dt, double dscale, const double* __restrict__ x0,
                                          const double* __restrict__ a0, double* __restrict__ x1,
                                          double* __restrict__ a1) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        for (int j = 0; j < d; ++j) {
            double v = 0.0, g = 0.0;
            for (int k = 0; k < split; ++k) {
                v += part[((long long)k * n + i) * dout + j];
                g += part[((long long)k * n + i) * dout + dout / 2 + j];
            }
            x1[i * d + j] = x0[i * d + j] + dt * v;
            if (a1 != nullptr) a1[i * d + j] = a0[i * d + j] - dt * (dscale * g);
        }
    }
}

struct EPDArgs {
    const double* x0;
    long long n;
    int d;
    const double* a0;
    int T;
    double sigma;
    int order;
    double* xt;
    double* at;
};

template <class Real, int KIND, int PDEG, int QDEG, int D>
int epd_impl(const EPDArgs& a, Workspace& ws, cudaStream_t st) {
    using Op = OpEPDiff<Real, KIND, PDEG, QDEG, D>;
    const SinglePlan pl = plan_single<Op>(a.n, a.n);
    float4* tgt = ws.take<float4>((size_t)Op::NS * pl.n_tpad);
    float4* src = ws.take<float4>((size_t)Op::NS * pl.m_pad);
    double* part = ws.take<double>((size_t)pl.split * a.n * Op::NOUT);
    double* center = ws.take<double>(kCenterWords);
    if (ws.measuring()) return LDDMM_OK;
    const KScale ks = kernel_scale(KIND, a.order, a.sigma, !pl.seq);
    typename Op::Params P{};
    P.src4 = src;
    P.src_stride = pl.m_pad;
    P.tgt4 = tgt;
    P.tgt_stride = pl.n_tpad;
    for (int j = 0; j < 5; ++j) P.pk[j] = (Real)ks.pk[j];
    for (int j = 0; j < 4; ++j) P.pq[j] = (Real)ks.pq[j];
    const long long N = a.n * a.d;
    const double dt = 1.0 / a.T;
    LDDMM_TRY(cuda_check(cudaMemcpyAsync(a.xt, a.x0, sizeof(double) * N, cudaMemcpyDeviceToDevice, st), "epdiff"));
    LDDMM_TRY(cuda_check(cudaMemcpyAsync(a.at, a.a0, sizeof(double) * N, cudaMemcpyDeviceToDevice, st), "epdiff"));
    const int nb = combine_blocks(a.n);
    launch_bbox_center(a.x0, a.n, nullptr, 0, a.d, center, st);
    for (int t = 0; t < a.T; ++t) {
        epd_pack_kernel<Real><<<grid_for(std::max(pl.n_tpad, pl.m_pad)), 256, 0, st>>>(
            a.xt + t * N, a.at + t * N, a.n, a.d, ks.scale, center, tgt, pl.n_tpad, src, pl.m_pad, Op::PP, D,
            Op::NS);
        LDDMM_TRY(launch_single<Op>(pl, a.n, P, nullptr, part, st));
        epd_combine_kernel<Real><<<nb, kCombineThreads, 0, st>>>(part, a.n, a.d, Op::NOUT, pl.split, dt, ks.dscale,
                                                                 a.xt + t * N, a.at + t * N, a.xt + (t + 1) * N,
                                                                 t + 1 < a.T ? a.at + (t + 1) * N : nullptr);
    }
    return cuda_check(cudaGetLastError(), "epdiff");
}

template <class Real>
int epd_run(const EPDArgs& a, Workspace& ws, cudaStream_t st) {
    if (a.order == 0) {
        set_error("epdiff: the order-0 Laplacian kernel is not differentiable");
        return LDDMM_ERR_ARG;
    }
    auto go = [&](auto kind, auto pdeg, auto qdeg) {
        return dispatch_d(a.d, [&](auto D) {
            return epd_impl<Real, decltype(kind)::value, decltype(pdeg)::value, decltype(qdeg)::value,
                            decltype(D)::value>(a, ws, st);
        });
    };
    switch (a.order) {
        case 1: return go(IC<KLAP>{}, IC<1>{}, IC<0>{});
        case 2: return go(IC<KLAP>{}, IC<2>{}, IC<1>{});
        case 3: return go(IC<KLAP>{}, IC<3>{}, IC<2>{});
        case 4: return go(IC<KLAP>{}, IC<4>{}, IC<3>{});
        default: return go(IC<KGAUSS>{}, IC<0>{}, IC<0>{});
    }
}

// ---- entry helpers --------------------------------------------------------------
static int basic_validate(long long n, int d, int T, double sigma, int order, const char* who) {
    if (n < 1 || n > (1LL << 30) || d < 1 || d > 3 || T < 1 || T > 100000 || !(sigma > 0) || order < 0) {
        set_error("%s: invalid arguments (n=%lld d=%d T=%d sigma=%g order=%d); d must be 1..3", who, n, d, T, sigma,
                  order);
        return LDDMM_ERR_ARG;
    }
    return LDDMM_OK;
}

template <class Run, class Args>
int run_with_workspace(Run run, const Args& a, void* wsp, size_t wsb, cudaStream_t st, const char* who) {
    Workspace meas;
    LDDMM_TRY(run(a, meas, st));
    if (wsp == nullptr || meas.off > wsb) {
        set_error("%s: workspace too small: need %zu bytes, got %zu", who, meas.off, wsb);
        return LDDMM_ERR_WORKSPACE;
    }
    LDDMM_TRY(check_device_ptr(wsp, "workspace"));
    Workspace ws;
    ws.base = static_cast<char*>(wsp);
    ws.cap = wsb;
    return run(a, ws, st);
}

template <class Real>
size_t shoot_ws(int64_t n, int d, int T, int nbatch = 1) {
    if (basic_validate(n, d, T, 1.0, 10, "shoot") != LDDMM_OK) return 0;
    if (nbatch < 1 || nbatch > kMaxBatch) return 0;
    ShootArgs a{};
    a.n = n;
    a.d = d;
    a.T = T;
    a.sigma = 1.0;
    a.order = 10;
    a.nbatch = nbatch;
    Workspace ws;
    size_t best = 0;
    for (int order : {10, 3}) {  // the Laplacian and Gaussian plans may differ
        a.order = order;
        ws = Workspace();
        shoot_run<Real>(a, ws, 0);
        best = std::max(best, ws.off);
    }
    return best + 256;
}

template <class Real>
int shoot_entry(const ShootArgs& a, void* wsp, size_t wsb, cudaStream_t st) {
    LDDMM_TRY(basic_validate(a.n, a.d, a.T, a.sigma, a.order, "shoot"));
    LDDMM_TRY(check_device_ptr(a.x0, "x0"));
    LDDMM_TRY(check_device_ptr(a.at, "at"));
    LDDMM_TRY(check_device_ptr(a.xt, "xt"));
    if (a.energy) LDDMM_TRY(check_device_ptr(a.energy, "energy"));
    if (a.dir != nullptr || a.eps != nullptr || a.at_try != nullptr || a.nbatch != 1) {
        if (a.nbatch < 1 || a.nbatch > kMaxBatch) {
            set_error("shoot: nbatch must be in [1, %d] (got %d)", kMaxBatch, a.nbatch);
            return LDDMM_ERR_ARG;
        }
        LDDMM_TRY(check_device_ptr(a.dir, "dir"));
        LDDMM_TRY(check_device_ptr(a.eps, "eps"));
        LDDMM_TRY(check_device_ptr(a.at_try, "at_try"));
    }
    return run_with_workspace([](const ShootArgs& q, Workspace& w, cudaStream_t s) { return shoot_run<Real>(q, w, s); },
                              a, wsp, wsb, st, "shoot");
}

template <class Real>
size_t cov_ws(int64_t n, int d, int T) {
    if (basic_validate(n, d, T, 1.0, 10, "covector") != LDDMM_OK) return 0;
    CovArgs a{};
    a.n = n;
    a.d = d;
    a.T = T;
    a.sigma = 1.0;
    size_t best = 0;
    for (int order : {10, 3}) {
        a.order = order;
        Workspace ws;
        cov_run<Real>(a, ws, 0);
        best = std::max(best, ws.off);
    }
    return best + 256;
}

template <class Real>
int cov_entry(const CovArgs& a, void* wsp, size_t wsb, cudaStream_t st) {
    LDDMM_TRY(basic_validate(a.n, a.d, a.T, a.sigma, a.order, "covector"));
    if (a.order == 0) {
        set_error("covector: the order-0 Laplacian kernel is not differentiable");
        return LDDMM_ERR_ARG;
    }
    LDDMM_TRY(check_device_ptr(a.xt, "xt"));
    LDDMM_TRY(check_device_ptr(a.at, "at"));
    LDDMM_TRY(check_device_ptr(a.px1, "px1"));
    LDDMM_TRY(check_device_ptr(a.pxt, "pxt"));
    if (a.dat) LDDMM_TRY(check_device_ptr(a.dat, "dat"));
    return run_with_workspace([](const CovArgs& q, Workspace& w, cudaStream_t s) { return cov_run<Real>(q, w, s); },
                              a, wsp, wsb, st, "covector");
}

template <class Real>
size_t epd_ws(int64_t n, int d, int T) {
    if (basic_validate(n, d, T, 1.0, 10, "epdiff") != LDDMM_OK) return 0;
    EPDArgs a{};
    a.n = n;
    a.d = d;
    a.T = T;
    a.sigma = 1.0;
    size_t best = 0;
    for (int order : {10, 3}) {
        a.order = order;
        Workspace ws;
        epd_run<Real>(a, ws, 0);
        best = std::max(best, ws.off);
    }
    return best + 256;
}

template <class Real>
int epd_entry(const EPDArgs& a, void* wsp, size_t wsb, cudaStream_t st) {
    LDDMM_TRY(basic_validate(a.n, a.d, a.T, a.sigma, a.order, "epdiff"));
    LDDMM_TRY(check_device_ptr(a.x0, "x0"));
    LDDMM_TRY(check_device_ptr(a.a0, "a0"));
    LDDMM_TRY(check_device_ptr(a.xt, "xt"));
    LDDMM_TRY(check_device_ptr(a.at, "at"));
    return run_with_workspace([](const EPDArgs& q, Workspace& w, cudaStream_t s) { return epd_run<Real>(q, w, s); },
                              a, wsp, wsb, st, "epdiff");
}

}  // namespace lddmm

using namespace lddmm;

extern "C" {

size_t lddmm_shoot_f32c_workspace(int64_t n, int d, int T) { return shoot_ws<float>(n, d, T); }
size_t lddmm_shoot_f64_workspace(int64_t n, int d, int T) { return shoot_ws<double>(n, d, T); }

int lddmm_shoot_f32c(const double* x0, int64_t n, int d, const double* at, int T, double dt, double sigma,
                     int order, double regweight, double* xt, double* energy, void* workspace,
                     size_t workspace_bytes, lddmm_stream_t stream) {
    ShootArgs a{x0, n, d, at, T, dt, sigma, order, regweight, xt, energy};
    return shoot_entry<float>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

int lddmm_shoot_f64(const double* x0, int64_t n, int d, const double* at, int T, double dt, double sigma,
                    int order, double regweight, double* xt, double* energy, void* workspace,
                    size_t workspace_bytes, lddmm_stream_t stream) {
    ShootArgs a{x0, n, d, at, T, dt, sigma, order, regweight, xt, energy};
    return shoot_entry<double>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

int lddmm_shoot_along_f32c(const double* x0, int64_t n, int d, const double* at, const double* dir, const double* eps,
                           int T, double dt, double sigma, int order, double regweight, double* at_try, double* xt,
                           double* energy, void* workspace, size_t workspace_bytes, lddmm_stream_t stream) {
    ShootArgs a{x0, n, d, at, T, dt, sigma, order, regweight, xt, energy};
    a.dir = dir;
    a.eps = eps;
    a.at_try = at_try;
    return shoot_entry<float>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

int lddmm_shoot_along_f64(const double* x0, int64_t n, int d, const double* at, const double* dir, const double* eps,
                          int T, double dt, double sigma, int order, double regweight, double* at_try, double* xt,
                          double* energy, void* workspace, size_t workspace_bytes, lddmm_stream_t stream) {
    ShootArgs a{x0, n, d, at, T, dt, sigma, order, regweight, xt, energy};
    a.dir = dir;
    a.eps = eps;
    a.at_try = at_try;
    return shoot_entry<double>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

size_t lddmm_shoot_along_batch_f32c_workspace(int64_t n, int d, int T, int nbatch) {
    return shoot_ws<float>(n, d, T, nbatch);
}
size_t lddmm_shoot_along_batch_f64_workspace(int64_t n, int d, int T, int nbatch) {
    return shoot_ws<double>(n, d, T, nbatch);
}

int lddmm_shoot_along_batch_f32c(const double* x0, int64_t n, int d, const double* at, const double* dir,
                                 const double* eps, int nbatch, int T, double dt, double sigma, int order,
                                 double regweight, double* at_try, double* xt, double* energy, void* workspace,
                                 size_t workspace_bytes, lddmm_stream_t stream) {
    ShootArgs a{x0, n, d, at, T, dt, sigma, order, regweight, xt, energy};
    a.dir = dir;
    a.eps = eps;
    a.at_try = at_try;
    a.nbatch = nbatch;
    return shoot_entry<float>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

int lddmm_shoot_along_batch_f64(const double* x0, int64_t n, int d, const double* at, const double* dir,
                                const double* eps, int nbatch, int T, double dt, double sigma, int order,
                                double regweight, double* at_try, double* xt, double* energy, void* workspace,
                                size_t workspace_bytes, lddmm_stream_t stream) {
    ShootArgs a{x0, n, d, at, T, dt, sigma, order, regweight, xt, energy};
    a.dir = dir;
    a.eps = eps;
    a.at_try = at_try;
    a.nbatch = nbatch;
    return shoot_entry<double>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

int lddmm_trial_batch_size(int64_t n, int d, int64_t nc, int64_t nc2, int shot_fp64, int value_fp64) {
    if (n < 1 || d < 2 || d > 3 || n > kFusedMaxPoints || !dt_fused_fits(nc, nc2)) return 1;
    // clusters of the batched shot and value kernels resident at once (the Gaussian
    // instances stand for the kernel family)
    auto shot = [&](auto D) {
        constexpr int D_ = decltype(D)::value;
        const FusedShape fs = fused_shape(n);
        return shot_fp64 ? fused_resident_clusters(shoot_fused_kernel<double, KGAUSS, 0, D_>, fs,
                                                   fused_dyn_smem<double>(n, D_), fused_dyn_smem<double>(kFusedMaxPoints, 3))
                         : fused_resident_clusters(shoot_fused_kernel<float, KGAUSS, 0, D_>, fs,
                                                   fused_dyn_smem<float>(n, D_), fused_dyn_smem<float>(kFusedMaxPoints, 3));
    };
    const int c = std::min(d == 2 ? shot(IC<2>{}) : shot(IC<3>{}), dt_value_resident_clusters(nc, nc2, d, value_fp64));
    return std::max(1, std::min(kTrialBatch, c));
}

size_t lddmm_covector_f32c_workspace(int64_t n, int d, int T) { return cov_ws<float>(n, d, T); }
size_t lddmm_covector_f64_workspace(int64_t n, int d, int T) { return cov_ws<double>(n, d, T); }

int lddmm_covector_f32c(const double* xt, int64_t n, int d, const double* at, int T, double dt, const double* px1,
                        double sigma, int order, double regweight, double* pxt, double* dat, void* workspace,
                        size_t workspace_bytes, lddmm_stream_t stream) {
    CovArgs a{xt, n, d, at, T, dt, px1, sigma, order, regweight, pxt, dat};
    return cov_entry<float>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

int lddmm_covector_f64(const double* xt, int64_t n, int d, const double* at, int T, double dt, const double* px1,
                       double sigma, int order, double regweight, double* pxt, double* dat, void* workspace,
                       size_t workspace_bytes, lddmm_stream_t stream) {
    CovArgs a{xt, n, d, at, T, dt, px1, sigma, order, regweight, pxt, dat};
    return cov_entry<double>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

size_t lddmm_epdiff_f32c_workspace(int64_t n, int d, int T) { return epd_ws<float>(n, d, T); }
size_t lddmm_epdiff_f64_workspace(int64_t n, int d, int T) { return epd_ws<double>(n, d, T); }

int lddmm_epdiff_f32c(const double* x0, int64_t n, int d, const double* a0, int T, double sigma, int order,
                      double* xt, double* at, void* workspace, size_t workspace_bytes, lddmm_stream_t stream) {
    EPDArgs a{x0, n, d, a0, T, sigma, order, xt, at};
    return epd_entry<float>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

int lddmm_epdiff_f64(const double* x0, int64_t n, int d, const double* a0, int T, double sigma, int order,
                     double* xt, double* at, void* workspace, size_t workspace_bytes, lddmm_stream_t stream) {
    EPDArgs a{x0, n, d, a0, T, sigma, order, xt, at};
    return epd_entry<double>(a, workspace, workspace_bytes, (cudaStream_t)stream);
}

}  // extern "C"
