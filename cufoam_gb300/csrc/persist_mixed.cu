// persist_mixed.cu -- mixed-precision solves (mixed.cu's algorithm) as one
// cooperative launch: the FP64 normFactor and residual, every FP32 sweep,
// the FP64 corrections and residuals, and the decisions between sweeps.
//
// The multi-kernel form spends a kernel boundary per pass (4 to 8 us) and a
// host round trip per sweep, and reads the FP32 matrix from HBM with an
// evict-first hint.  Here a pass boundary is a grid barrier (1.2 us) or sum
// (2.5 us), nothing returns to the host, and a matrix that fits in L2 beside
// the vectors stays there.  The search direction is formed in its own pass
// and gathered once per entry (the multi-kernel CG and BiCGStab passes form
// it for every gathered entry to save a kernel).  Dot products: FP32 products
// and FP32 sums per thread, as before, the threads' sums in fixed point and
// FP64 (more exact than FP32 trees).
//
// us per FP32 step, multi-kernel form -> here (7-point systems; set-up of a
// solve 149 -> 43 us at 22k rows, 511 -> 233 at 2.1M):
//              22k          219k          893k          2.1M rows
//   CG         15.5-> 8.0   25.7->10.3   36.1->17.2   52.9->34.7
//   MR         10.0-> 6.9   17.1-> 8.7   23.4->13.9   33.7->27.3
//   BiCGStab   27.0->15.6   51.4->20.4   68.4->37.9   91.2->73.1
// At 2.1M rows a CG step moves about 110 MB through L2 (5 bytes per slot and
// the vectors); latency and the 64-register budget bound it.
#include "persist.cuh"

#include <algorithm>
#include <climits>
#include <cstring>

namespace cf {

enum { kMxCG = 0, kMxMR = 1, kMxBCS = 2 };

// byte offsets of the block-private FP32 vectors and the block's matrix
// slots in dynamic shared memory (-1: in global memory)
struct MixedPlan {
    int32_t r, q, d, own, own2, t, rh;
    int32_t val, col, off;
};

struct MixedArgs {
    PersistGrid g;
    DevState *out;           // host-mapped: the final FP64 state
    DevState *out_in;        // host-mapped: k = total FP32 steps
    double tolerance, rel_tol, eta;
    long long max_total;
    int32_t max_steps, min_steps, max_outer, inner_cap, hist_cap, abs_tol, l1;
    int32_t jmr;             // the residual is D^-1/2 (b - A x)
    int32_t keep;            // the FP32 matrix fits in L2: no evict-first hint
    double *x_keep, *r_keep; // x and r before a correction
    const int32_t *first;    // streamed: the blocks' first slices (null: equal numbers)
    MixedPlan plan;
};

struct MixedState {
    // FP64 refinement
    double tol, nf, norm, norm0, xbar, prev;
    long long total;
    int32_t k, done, status, result, cap, stop;
    // FP32 sweep
    float rho0, rho1, xi, omega, theta, tol_in;
    int32_t k_in, done_in, status_in, max_in;
};

template <int FMT> struct MixedCols;
template <> struct MixedCols<kSell> {
    static __device__ __forceinline__ SellCols32 make(const SolveArgs &A) { return SellCols32{A.s_col}; }
};
template <> struct MixedCols<kSellC> {
    static __device__ __forceinline__ SellCodes8 make(const SolveArgs &A) { return SellCodes8(A.s_code, A.s_dtab); }
};
template <> struct MixedCols<kSellD> {
    static __device__ __forceinline__ SellDelta16 make(const SolveArgs &A) { return SellDelta16{A.s_d16}; }
};

// the block's rows, four slices (s, s + nw, ...) per round: a pass loads into
// arrays indexed by h in one CF_MX_EACH loop and stores in a second
#define CF_MX_ROUNDS(s) for (int s = s_lo + warp; s < s_hi; s += 4 * nw)
#define CF_MX_EACH(s, h, row, i)                                                          \
    _Pragma("unroll") for (int h = 0; h < 4; ++h)                                        \
        if (const int row = 32 * (s + h * nw) + lane, i = row - base; s + h * nw < s_hi && row < n && i >= 0)

template <int SOLVER, int FMT, bool LOCALM, class SYNC>
__global__ void __launch_bounds__(SYNC::kThreads, 1)
    k_persist_mixed(const __grid_constant__ SolveArgs A, const __grid_constant__ MixedArgs P)
{
    __shared__ typename SYNC::Shared sh;
    __shared__ MixedState st;
    extern __shared__ __align__(16) unsigned char smem_[];
    if (threadIdx.x == 0) {
        st = MixedState{};
        st.k = -1;   // (no residual yet)
    }
    SYNC gs(P.g, &sh);

    const int n = A.n, ns = A.n_slices;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int rank = gs.rank();
    const bool first = rank == 0;
    const bool table = !LOCALM && P.first;
    const int s_lo = table ? P.first[rank] : (int)((int64_t)ns * rank / gs.blocks());
    const int s_hi = table ? P.first[rank + 1] : (int)((int64_t)ns * (rank + 1) / gs.blocks());
    const int base = 32 * s_lo;
    const uint64_t pol = P.keep ? l2_evict_normal_policy() : l2_evict_first_policy();
    const uint64_t pol64 = l2_evict_first_policy();
    const auto cols = MixedCols<FMT>::make(A);
    const bool has_long = A.has_long != 0;
    double *const x = A.x;
    const double *const b = A.b;
    double *const r64 = A.r[0];
    auto at = [&](int32_t o, float *global) {
        return LOCALM || o >= 0 ? reinterpret_cast<float *>(smem_ + o) : global + base;
    };
    // gathered: p (CG, BiCGStab), r (MR), s (BiCGStab)
    float *const gv = SOLVER == kMxMR ? A.fr : A.fp[0];
    float *const gs2 = A.fp[1];
    float *const rl = at(P.plan.r, A.fr);            // own r
    float *const q = at(P.plan.q, A.fq);             // q, y or v
    float *const d = at(P.plan.d, A.fx);             // the correction
    float *const own = SOLVER == kMxMR ? rl : at(P.plan.own, A.fp[0]);
    float *const own2 = at(P.plan.own2, A.fp[1]);
    float *const t = at(P.plan.t, A.fqs);
    float *const rh = at(P.plan.rh, A.frs);
    float *const rg = SOLVER == kMxMR && rl != A.fr + base ? A.fr + base : nullptr;
    const int32_t *off = A.s_off + s_lo;
    const float *lval = nullptr;
    const int32_t *lcol = nullptr;
    if (LOCALM || P.plan.off >= 0) {
        int32_t *o = reinterpret_cast<int32_t *>(smem_ + P.plan.off);
        for (int s = threadIdx.x; s <= s_hi - s_lo; s += blockDim.x) o[s] = A.s_off[s_lo + s];
        off = o;
    }
    if constexpr (LOCALM) {
        const int e0 = A.s_off[s_lo], e1 = A.s_off[s_hi];
        float *dv = reinterpret_cast<float *>(smem_ + P.plan.val);
        int32_t *dc = reinterpret_cast<int32_t *>(smem_ + P.plan.col);
        for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
            dv[e - e0] = __ldg(A.s_val32 + e);
            dc[e - e0] = __ldg(A.s_col + e);
        }
        lval = dv;
        lcol = dc;
    }
    __syncthreads();

    auto product = [&](int s, const float *v) {
        const int o = off[s - s_lo], len = (off[s - s_lo + 1] - o) >> 5;
        auto g = [&](int c) { return v[c]; };
        if constexpr (LOCALM) {
            const int l = o - off[0] + lane;
            return local_slice<float, kSellBatch32>(lcol + l, lval + l, len, g);
        } else {
            return sell_slice_at<float, kSellBatch32>(n, s, o, len, cols, A.s_val32, A.ro, has_long, pol, g);
        }
    };
    auto product64 = [&](int s, auto g) {
        const int o = off[s - s_lo], len = (off[s - s_lo + 1] - o) >> 5;
        return sell_slice_at<double, kSellBatch>(n, s, o, len, cols, A.s_val, A.ro, has_long, pol64, g);
    };
    auto record = [&](int k, double norm) {
        if (first && k < P.hist_cap) {
            if (A.hist) A.hist[k] = norm;
            if (A.hist_t) A.hist_t[k] = global_ns();
        }
    };
    // after a step of a sweep: the stopping rules of finish_step
    auto step_in = [&](float rr, bool stop) {
        const float norm = sqrtf(rr);
        const int k = st.k_in + 1;
        st.k_in = k;
        const bool finite = isfinite(norm);
        const bool cont = finite && k < st.max_in && norm > st.tol_in && !stop;
        st.status_in = stop ? CF_TIMEOUT : !finite ? CF_NONFINITE : (norm > st.tol_in ? CF_NOT_CONVERGED : CF_OK);
        st.done_in = cont ? 0 : 1;
        if (stop) st.stop = 1;
    };

    // ---- FP64 normFactor and initial residual ------------------------------
    {
        double acc[1] = {0.0};
        for (int s = s_lo + warp; s < s_hi; s += nw) {
            const int row = 32 * s + lane;
            if (row < n) acc[0] += x[row];
        }
        if (!gs.sum(acc, nullptr, [&](const double(&v)[1]) { st.xbar = v[0] / n; })) goto out;
    }
    {
        const double xbar = st.xbar;
        const double cval = P.l1 ? 1.0 : xbar;
        double acc[3] = {0.0, 0.0, 0.0};
        for (int s = s_lo + warp; s < s_hi; s += nw) {
            const int row = 32 * s + lane;
            const double y = product64(s, [&](int c) { return x[c]; });
            double yb = product64(s, [&](int) { return cval; });
            if (P.l1) yb = __dmul_rn(yb, xbar);
            if (row < n) {
                const double bi = b[row];
                const double d1 = y - yb, d2 = bi - yb;
                double ri = bi - y;
                if (P.jmr) ri = __dmul_rn(A.dinv_sqrt[row], ri);
                r64[row] = ri;
                if (P.l1) {
                    acc[0] += fabs(d1) + fabs(d2);
                } else {
                    acc[0] = fma_t(d1, d1, acc[0]);
                    acc[1] = fma_t(d2, d2, acc[1]);
                }
                acc[2] = fma_t(ri, ri, acc[2]);
            }
        }
        if (!gs.sum(acc, nullptr, [&](const double(&v)[3]) {
                const double nf = P.l1 ? v[0] + 1e-20 : sqrt(v[0]) + sqrt(v[1]) + 1e-20;
                const double norm0 = sqrt(v[2]);
                st.nf = nf;
                st.tol = P.abs_tol ? P.tolerance : P.tolerance * nf;
                if (P.rel_tol > 0.0) st.tol = fmax(st.tol, P.rel_tol * norm0);
                st.norm = st.norm0 = norm0;
                record(0, norm0);
                const bool finite = isfinite(norm0);
                const bool cont = finite && P.max_steps >= 1 && (norm0 > st.tol || P.min_steps > 0);
                st.done = cont ? 0 : 1;
                st.status = !finite ? CF_NONFINITE : (norm0 > st.tol ? CF_NOT_CONVERGED : CF_OK);
                st.result = st.done ? st.status : CF_NOT_CONVERGED;
                st.k = 0;
                st.total = 0;
                st.prev = norm0;
                st.cap = P.inner_cap;
                st.stop = 0;
            }))
            goto out;
    }

    // ---- refinement sweeps -------------------------------------------------
    for (int outer = 0; !st.done && outer < P.max_outer && st.total < P.max_total && !st.stop; ++outer) {
        // r32 = r64 / ||r64||, d = 0
        {
            const double inv = 1.0 / st.norm;
            float acc = 0.f;
            for (int s = s_lo + warp; s < s_hi; s += nw) {
                const int row = 32 * s + lane, i = row - base;
                if (row < n) {
                    const float v = (float)(r64[row] * inv);
                    rl[i] = v;
                    if (rg) rg[i] = v;
                    d[i] = 0.f;
                    if (SOLVER == kMxBCS) rh[i] = v;
                    acc = fma_t(v, v, acc);
                }
            }
            const double a1[1] = {(double)acc};
            if (!gs.sum(a1, nullptr, [&](const double(&v)[1]) {
                    const float rr = (float)v[0];
                    const float norm0 = sqrtf(rr);
                    // the last sweep only has to reach the FP64 target
                    const double rtol = fmax(P.eta, fmin(0.5, 0.8 * st.tol / st.prev));
                    st.rho0 = rr;
                    st.rho1 = 0.f;
                    st.xi = st.omega = st.theta = 0.f;
                    st.tol_in = (float)(rtol * norm0);
                    st.k_in = 0;
                    const long long left = P.max_total - st.total;
                    st.max_in = (int)(left < st.cap ? left : st.cap);
                    const bool finite = isfinite(norm0);
                    const bool cont = finite && st.max_in >= 1 && (SOLVER == kMxBCS || norm0 > st.tol_in);
                    st.done_in = cont ? 0 : 1;
                    st.status_in = finite ? CF_OK : CF_NONFINITE;
                }))
                goto out;
        }
        for (int k = 1; !st.done_in; ++k) {
            if constexpr (SOLVER == kMxCG) {
                // d += xi p (the previous step), p = r + beta p
                const float beta = k == 1 ? 0.f : st.rho0 / st.rho1, xi = st.xi;
                CF_MX_ROUNDS(s) {
                    float pv[4], dv[4], rv[4];
                    CF_MX_EACH(s, h, row, i) {
                        rv[h] = rl[i];
                        if (k > 1) {
                            pv[h] = own[i];
                            dv[h] = d[i];
                        }
                    }
                    CF_MX_EACH(s, h, row, i) {
                        if (k > 1) {
                            d[i] = fma_t(xi, pv[h], dv[h]);
                            rv[h] = fma_t(beta, pv[h], rv[h]);
                        }
                        gv[row] = rv[h];
                        if (LOCALM) own[i] = rv[h];
                    }
                }
                if (!gs.barrier()) goto out;
                float acc = 0.f;
                for (int s = s_lo + warp; s < s_hi; s += nw) {
                    const int row = 32 * s + lane, i = row - base;
                    const float y = product(s, gv);
                    if (row < n) {
                        q[i] = y;
                        acc = fma_t(own[i], y, acc);
                    }
                }
                const double a1[1] = {(double)acc};
                if (!gs.sum(a1, nullptr, [&](const double(&v)[1]) { st.xi = st.rho0 / (float)v[0]; })) goto out;
                const float al = st.xi;
                float rr = 0.f;
                CF_MX_ROUNDS(s) {
                    float qv[4], rv[4];
                    CF_MX_EACH(s, h, row, i) {
                        qv[h] = q[i];
                        rv[h] = rl[i];
                    }
                    CF_MX_EACH(s, h, row, i) {
                        const float ri = fma_t(-al, qv[h], rv[h]);
                        rl[i] = ri;
                        rr = fma_t(ri, ri, rr);
                    }
                }
                const double a2[1] = {(double)rr};
                if (!gs.sum(a2, A.abort_flag, [&](const double(&v)[1]) {
                        st.rho1 = st.rho0;
                        st.rho0 = (float)v[0];
                        step_in((float)v[0], sh.stop != 0);
                    }))
                    goto out;
            } else if constexpr (SOLVER == kMxMR) {
                float a0 = 0.f, a1 = 0.f;
                for (int s = s_lo + warp; s < s_hi; s += nw) {
                    const int row = 32 * s + lane, i = row - base;
                    const float y = product(s, gv);
                    if (row < n) {
                        q[i] = y;
                        a0 = fma_t(own[i], y, a0);
                        a1 = fma_t(y, y, a1);
                    }
                }
                const double av[2] = {(double)a0, (double)a1};
                if (!gs.sum(av, nullptr, [&](const double(&v)[2]) { st.omega = (float)v[0] / (float)v[1]; })) goto out;
                const float w = st.omega;
                float rr = 0.f;
                CF_MX_ROUNDS(s) {
                    float yv[4], rv[4], dv[4];
                    CF_MX_EACH(s, h, row, i) {
                        yv[h] = q[i];
                        rv[h] = rl[i];
                        dv[h] = d[i];
                    }
                    CF_MX_EACH(s, h, row, i) {
                        d[i] = fma_t(w, rv[h], dv[h]);
                        const float ri = fma_t(-w, yv[h], rv[h]);
                        rl[i] = ri;
                        if (rg) rg[i] = ri;
                        rr = fma_t(ri, ri, rr);
                    }
                }
                const double a2[1] = {(double)rr};
                if (!gs.sum(a2, A.abort_flag,
                            [&](const double(&v)[1]) { step_in((float)v[0], sh.stop != 0); }))
                    goto out;
            } else {
                // BiCGStab: p = r + beta (p - omega v)
                const float beta = st.theta, w0 = st.omega;
                CF_MX_ROUNDS(s) {
                    float pv[4], vv[4], rv[4];
                    CF_MX_EACH(s, h, row, i) {
                        rv[h] = rl[i];
                        if (k > 1) {
                            pv[h] = own[i];
                            vv[h] = q[i];
                        }
                    }
                    CF_MX_EACH(s, h, row, i) {
                        if (k > 1) rv[h] = fma_t(beta, fma_t(-w0, vv[h], pv[h]), rv[h]);
                        gv[row] = rv[h];
                        if (LOCALM) own[i] = rv[h];
                    }
                }
                if (!gs.barrier()) goto out;
                // v = A p, alpha = rho / (r^, v)
                float acc = 0.f;
                for (int s = s_lo + warp; s < s_hi; s += nw) {
                    const int row = 32 * s + lane, i = row - base;
                    const float y = product(s, gv);
                    if (row < n) {
                        q[i] = y;
                        acc = fma_t(rh[i], y, acc);
                    }
                }
                const double a1[1] = {(double)acc};
                if (!gs.sum(a1, nullptr, [&](const double(&v)[1]) {
                        const float tot = (float)v[0], alpha = st.rho0 / tot;
                        if (isfinite(alpha) && tot != 0.f) {
                            st.xi = alpha;
                        } else {
                            st.done_in = 1;
                            st.status_in = tot == 0.f ? CF_BREAKDOWN : CF_NONFINITE;
                        }
                    }))
                    goto out;
                if (st.done_in) break;
                const float alpha = st.xi;
                // s = r - alpha v
                CF_MX_ROUNDS(s) {
                    float vv[4], rv[4];
                    CF_MX_EACH(s, h, row, i) {
                        vv[h] = q[i];
                        rv[h] = rl[i];
                    }
                    CF_MX_EACH(s, h, row, i) {
                        const float si = fma_t(-alpha, vv[h], rv[h]);
                        gs2[row] = si;
                        if (LOCALM) own2[i] = si;
                    }
                }
                if (!gs.barrier()) goto out;
                // t = A s, omega = (t, s) / (t, t)
                float b0 = 0.f, b1 = 0.f;
                for (int s = s_lo + warp; s < s_hi; s += nw) {
                    const int row = 32 * s + lane, i = row - base;
                    const float y = product(s, gs2);
                    if (row < n) {
                        t[i] = y;
                        b0 = fma_t(y, own2[i], b0);
                        b1 = fma_t(y, y, b1);
                    }
                }
                const double bv[2] = {(double)b0, (double)b1};
                if (!gs.sum(bv, nullptr, [&](const double(&v)[2]) {
                        const float t1 = (float)v[1];
                        st.omega = t1 > 0.f ? (float)v[0] / t1 : 0.f;
                    }))
                    goto out;
                // d += alpha p + omega s, r = s - omega t, ||r||, (r^, r)
                const float w = st.omega;
                float c0 = 0.f, c1 = 0.f;
                CF_MX_ROUNDS(s) {
                    float sv[4], tv[4], dv[4], pv[4], hv[4];
                    CF_MX_EACH(s, h, row, i) {
                        sv[h] = own2[i];
                        tv[h] = t[i];
                        dv[h] = d[i];
                        pv[h] = own[i];
                        hv[h] = rh[i];
                    }
                    CF_MX_EACH(s, h, row, i) {
                        d[i] = fma_t(w, sv[h], fma_t(alpha, pv[h], dv[h]));
                        const float ri = fma_t(-w, tv[h], sv[h]);
                        rl[i] = ri;
                        c0 = fma_t(ri, ri, c0);
                        c1 = fma_t(hv[h], ri, c1);
                    }
                }
                const double cv[2] = {(double)c0, (double)c1};
                if (!gs.sum(cv, A.abort_flag, [&](const double(&v)[2]) {
                        const float norm = sqrtf((float)v[0]), rho = (float)v[1];
                        const int kk = st.k_in + 1;
                        st.k_in = kk;
                        bool cont = true;
                        int status = CF_NOT_CONVERGED;
                        if (norm < st.tol_in) {
                            cont = false;
                            status = CF_OK;
                        } else if (kk >= st.max_in) {
                            cont = false;
                        } else if (!isfinite(norm)) {
                            cont = false;
                            status = CF_NONFINITE;
                        } else if (rho == 0.f || w == 0.f) {
                            cont = false;
                            status = CF_BREAKDOWN;
                        }
                        if (sh.stop) {
                            cont = false;
                            status = CF_TIMEOUT;
                            st.stop = 1;
                        }
                        if (cont) {
                            st.theta = (rho / st.rho0) * (alpha / w);
                            st.rho1 = st.rho0;
                            st.rho0 = rho;
                        } else {
                            st.done_in = 1;
                            st.status_in = status;
                        }
                    }))
                    goto out;
            }
        }
        // x and r kept, x += ||r|| d (MR family: ||r|| R d); the last CG step
        // still has to reach d
        {
            const double sc = st.norm;
            const float xi = st.xi;
            const bool last = SOLVER == kMxCG && st.k_in > 0;
            const double *R = A.corr_scale;
            for (int s = s_lo + warp; s < s_hi; s += nw) {
                const int row = 32 * s + lane, i = row - base;
                if (row < n) {
                    const float df = last ? fma_t(xi, own[i], d[i]) : d[i];
                    double di = (double)df;
                    if (R) di *= R[row];
                    const double x0 = x[row];
                    P.x_keep[row] = x0;
                    P.r_keep[row] = r64[row];
                    x[row] = fma_t(sc, di, x0);
                }
            }
            if (!gs.barrier()) goto out;
        }
        // FP64 residual, and the rules of the refinement loop
        {
            double acc[1] = {0.0};
            for (int s = s_lo + warp; s < s_hi; s += nw) {
                const int row = 32 * s + lane;
                const double y = product64(s, [&](int c) { return x[c]; });
                if (row < n) {
                    double ri = b[row] - y;
                    if (P.jmr) ri = __dmul_rn(A.dinv_sqrt[row], ri);
                    r64[row] = ri;
                    acc[0] = fma_t(ri, ri, acc[0]);
                }
            }
            if (!gs.sum(acc, nullptr, [&](const double(&v)[1]) {
                    const double norm = sqrt(v[0]);
                    st.k += 1;
                    record(st.k, norm);
                    st.total += st.k_in;
                    st.norm = norm;
                    if (isfinite(norm) && norm <= st.tol) {
                        st.done = 1;
                        st.status = st.result = CF_OK;
                    } else if (st.status_in == CF_BREAKDOWN && st.k_in == 0) {
                        // x is unchanged: a retry would break down again
                        st.done = 1;
                        st.status = isfinite(norm) ? CF_BREAKDOWN : CF_NONFINITE;
                        st.result = st.status;
                    } else if (!(norm < st.prev)) {
                        st.done = 2;   // undo, and retry half as long (below)
                    } else {
                        st.prev = norm;
                    }
                }))
                goto out;
        }
        if (st.done == 2) {
            for (int s = s_lo + warp; s < s_hi; s += nw) {
                const int row = 32 * s + lane;
                if (row < n) {
                    x[row] = P.x_keep[row];
                    r64[row] = P.r_keep[row];
                }
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                st.norm = st.prev;
                st.done = 0;
                st.status = CF_NOT_CONVERGED;
                st.cap = st.k_in / 2;
                if (st.cap < 8) st.done = 1;
                st.result = CF_NOT_CONVERGED;
            }
            __syncthreads();
        }
    }
out:
    if (first && threadIdx.x == 0) {
        DevState *o = P.out;
        o->nf = st.nf;
        o->norm0 = st.norm0;
        o->norm = st.norm;
        o->omega = 0.0;
        o->k = st.k;
        o->status = st.stop ? CF_TIMEOUT : st.result;
        P.out_in->k = (int32_t)(st.total < INT_MAX ? st.total : INT_MAX);
    }
    report_fail(sh.fail, P.out);
    gs.leave();
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
template <int SOLVER>
static const void *mixed_pick(int scope, int format)
{
    if (scope == kScopeCluster) return (const void *)k_persist_mixed<SOLVER, kSell, true, ClusterSync>;
    if (scope == kScopeGridLocal) return (const void *)k_persist_mixed<SOLVER, kSell, true, GridSync>;
    return format == kSellC   ? (const void *)k_persist_mixed<SOLVER, kSellC, false, GridSync>
           : format == kSellD ? (const void *)k_persist_mixed<SOLVER, kSellD, false, GridSync>
                              : (const void *)k_persist_mixed<SOLVER, kSell, false, GridSync>;
}

void launch_persist_mixed(Context *ctx, int solver, int format, const SolveArgs &A, const DevState &S, int l1,
                          Matrix *m, const cf_controls &c, DevState *out, DevState *out_in)
{
    const int max_len = m->sell_max_len;   // slots per row of the longest slice
    MixedArgs P;
    std::memset(&P, 0, sizeof(P));
    P.g = persist_grid(ctx);
    P.out = out;
    P.out_in = out_in;
    P.tolerance = S.tolerance;
    P.rel_tol = S.rel_tol;
    P.eta = mixed_inner_tolerance(c, solver);
    P.max_total = c.max_iter <= 0 ? INT_MAX : c.max_iter;
    P.max_steps = S.max_steps;
    P.min_steps = S.min_steps;
    P.max_outer = c.mixed_max_outer > 0 ? c.mixed_max_outer : 50;
    P.inner_cap = c.mixed_inner_max > 0 ? c.mixed_inner_max : INT_MAX;
    P.hist_cap = S.hist_cap;
    P.abs_tol = (S.flags & kFlagAbsTol) ? 1 : 0;
    P.l1 = l1;
    P.jmr = solver == CF_JMR ? 1 : 0;
    P.x_keep = A.w[0];
    P.r_keep = A.w[1];

    const int kind = solver == CF_CG ? kMxCG : solver == CF_BICG ? kMxBCS : kMxMR;
    const int ns = A.n_slices;
    auto plan = [&](int slices, bool matrix, size_t cap) {
        MixedPlan p;
        std::memset(&p, -1, sizeof(p));
        size_t at = 0;
        auto take = [&](bool want, size_t bytes) {
            if (!want || at + bytes > cap) return -1;
            const int32_t o = (int32_t)at;
            at += (bytes + 15) / 16 * 16;
            return o;
        };
        const size_t vec = sizeof(float) * 32 * (size_t)slices;
        p.off = take(slices <= 8192, sizeof(int32_t) * ((size_t)slices + 1));
        if (matrix) {
            p.val = take(true, vec * max_len);
            p.col = take(true, vec * max_len);
        }
        p.q = take(true, vec);
        p.r = take(matrix || kind != kMxMR, vec);
        p.d = take(true, vec);
        if (kind == kMxBCS) {
            p.rh = take(true, vec);
            p.t = take(true, vec);
        }
        if (matrix && kind != kMxMR) p.own = take(true, vec);
        if (matrix && kind == kMxBCS) p.own2 = take(true, vec);
        return std::make_pair(p, at);
    };
    auto complete = [&](const MixedPlan &p) {
        return p.off >= 0 && p.val >= 0 && p.col >= 0 && p.q >= 0 && p.r >= 0 && p.d >= 0 &&
               (kind == kMxMR || p.own >= 0) && (kind != kMxBCS || (p.rh >= 0 && p.t >= 0 && p.own2 >= 0));
    };
    int scope = kScopeGrid, grid = 1, most = 0;   // (most: slices of a block)
    size_t smem = 0;
    const bool small_rows = !A.has_long && max_len <= kLongRow;
    auto pick = [&](int in) {
        return kind == kMxCG   ? mixed_pick<kMxCG>(in, format)
               : kind == kMxMR ? mixed_pick<kMxMR>(in, format)
                               : mixed_pick<kMxBCS>(in, format);
    };
    if (small_rows && A.n <= CF_PERSIST_CLUSTER_ROWS && persist_cluster_fits(ctx, pick(kScopeCluster))) {
        while (grid < 16 && 4 * grid < ns) grid <<= 1;
        const auto pl = plan((ns + grid - 1) / grid, true, CF_PERSIST_LOCAL_BYTES - sizeof(ClusterSync::Shared));
        if (complete(pl.first)) {
            scope = kScopeCluster;
            P.plan = pl.first;
            smem = pl.second;
        }
    }
    if (scope == kScopeGrid) {
        grid = std::max(1, std::min(ctx->sm_count, (ns + 3) / 4));
        const int slices = (ns + grid - 1) / grid;
        auto pl = plan(slices, small_rows, CF_PERSIST_LOCAL_BYTES);
        if (small_rows && complete(pl.first)) {
            scope = kScopeGridLocal;
        } else {
            P.first = persist_shares(m, grid, most);
            pl = plan(most, false, CF_PERSIST_VEC_BYTES);
        }
        P.plan = pl.first;
        smem = pl.second;
    }
    const double slot = format == kSellC ? 5.0 : format == kSellD ? 6.0 : 8.0;
    P.keep = slot * (double)m->sell_nnz + 40.0 * A.n < 0.95 * (double)ctx->l2_bytes ? 1 : 0;
    const void *kernel = pick(scope);
    SolveArgs a = A;
    void *args[] = {&a, &P};
    out->flags = 0;   // (S may be *out: read above)
    launch_persist_kernel(ctx, kernel, scope == kScopeCluster, grid, most ? most : (ns + grid - 1) / grid, smem,
                          args);
}

} // namespace cf
