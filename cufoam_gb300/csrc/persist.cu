// persist.cu -- FP64 solves in the fast summation order as one cooperative
// launch: normFactor, the initial residual, every step and the last update
// of psi, with a grid barrier where the multi-kernel loop (solve_fast.cu)
// has a kernel boundary.
//
// What bounds the multi-kernel loop below about a million rows is not bytes
// or FP64 issue but its boundaries: launch, ramp-up, drain and the last
// block's serial reduction, 4 to 8 us per kernel.  A grid barrier costs 1.2
// us here, a grid sum about 2.5.
//
// Three forms, by size:
//   * up to CF_PERSIST_CLUSTER_ROWS one cluster of up to 16 blocks: hardware
//     barriers (0.5 us) and sums through distributed shared memory;
//   * the grid, with each block's matrix slots and vectors in shared memory
//     for the whole solve while they fit (about 250k rows of a 7-point
//     system): only the gathered vector is exchanged, through L2;
//   * the grid with the matrix streamed from L2 or HBM.
// Large systems, whose vectors outgrow L2, stay with the multi-kernel loop
// (persist_usable).
// Measured on GB300, us per step and for normFactor + residual + first step
// (7-point systems; multi-kernel loop, or the single-cluster kernels at 4k
// rows -> here):
//                4k          22k         219k        893k        2.1M rows
//   CG step      7.0->5.0   16.6->7.9   28.8->12.8  43.9->27.0  72.1->55.7
//   Jacobi step  4.7->2.2    8.3->3.4   15.3->7.4   28.8->20.6  53.5->43.9
//   MRJacobi     8.2->5.1   16.0->7.2   24.0->12.3  38.8->25.8  70.4->53.9
//   CG set-up     27->24     102->30     160->48     267->94     422->170
// At 2.1M rows the FP64 unit bounds a CG step: 12 operations per row, 64
// cycles per warp and sub-partition each, are 83,000 of its 115,000 cycles.
// The arithmetic of a row and of an element
// is the loop's: one FMA chain per row in entry order, one FMA per update;
// only how the dot products are summed differs.
#include "persist.cuh"

#include <algorithm>
#include <climits>
#include <cstring>
#include <type_traits>

namespace cf {

// Where a block keeps what only it reads, in doubles from the start of its
// dynamic shared memory (-1: in global memory).
struct PersistPlan {
    int32_t q, r, x, scale;  // y / q, own r, x, the diagonal scaling
    int32_t g;               // own rows of the gathered p or z (with the matrix only)
    int32_t g2;              // in a cluster: a second gathered vector (Jacobi's r, Richardson's power method)
    int32_t val, col;        // this block's slots of the loop's matrix
    int32_t off;             // its slices' offsets (always there)
};

struct PersistArgs {
    PersistGrid g;
    DevState *out;           // host-mapped: the final state
    double tolerance, rel_tol, omega, diag_abs_min;
    int32_t max_steps, min_steps, hist_cap;
    int32_t abs_tol, l1, power_steps;
    int32_t head;            // log2 of the rows per thread, and one (FixedDot)
    int32_t keep;            // the matrix fits in L2 beside the vectors: no evict-first hint
    const int32_t *first;    // streamed: the blocks' first slices (null: equal numbers)
    PersistPlan plan;
};

// Per-block step state, the same bits in every block (thread 0 writes it
// between barriers).
struct PersistState {
    double rho0, rrho, xi, beta, omega, tol, tol_hi, nf, norm, norm0, xbar, pow_inv, lambda;
    int32_t k, done, status;
};

// CF_CG, CF_PCG, CF_JACOBI, CF_RICHARDSON, CF_MR; MRJacobi and MRS run as
// CF_MRJACOBI (z = D^-1 r gathered), JMR as CF_JMR (MR on the scaled matrix)
template <int SOLVER> struct PersistTraits {
    static constexpr bool kCgLike = SOLVER == CF_CG || SOLVER == CF_PCG;
    static constexpr bool kMr = SOLVER == CF_MR || SOLVER == CF_MRJACOBI || SOLVER == CF_JMR;
    // r read by other blocks (gathered by the product)
    static constexpr bool kGatherR = SOLVER == CF_MR || SOLVER == CF_JMR || SOLVER == CF_JACOBI;
    static constexpr bool kQ = kCgLike || kMr;
    // a gathered vector whose own rows are read again: p, z
    static constexpr bool kOwnG = kCgLike || SOLVER == CF_MRJACOBI;
    static constexpr bool kLocalX = SOLVER != CF_RICHARDSON;   // (Richardson gathers x)
    static constexpr bool kScale = SOLVER == CF_PCG || SOLVER == CF_JACOBI || SOLVER == CF_MRJACOBI || SOLVER == CF_JMR;
    static constexpr bool kScaledMatrix = SOLVER == CF_JACOBI || SOLVER == CF_JMR;
};

__device__ __forceinline__ void persist_record(const SolveArgs &A, const PersistArgs &P, bool first, int k, double norm)
{
    if (first && k < P.hist_cap) {
        if (A.hist) A.hist[k] = norm;
        if (A.hist_t) A.hist_t[k] = global_ns();
    }
}

// after the initial residual (finish_init's rules)
__device__ __forceinline__ void persist_begin(const SolveArgs &A, const PersistArgs &P, bool first, PersistState &st,
                                              double rr)
{
    const double norm0 = sqrt(rr);
    st.rho0 = rr;
    st.norm0 = st.norm = norm0;
    persist_record(A, P, first, 0, norm0);
    if (P.rel_tol > 0.0) st.tol = fmax(st.tol, P.rel_tol * norm0);
    // ||r|| > tol is decided on (r, r) without the square root (about fifteen
    // dependent FP64 operations on the step's critical path) unless it is
    // within rounding of tol^2
    const double t2 = st.tol * st.tol;
    const bool usable = t2 > 1e-280 && t2 < 1e280;
    st.tol_hi = usable ? t2 * (1.0 + 1e-14) : HUGE_VAL;
    st.k = 0;
    const bool finite = isfinite(norm0);
    const bool cont = finite && P.max_steps >= 1 && (norm0 > st.tol || P.min_steps > 0);
    st.done = cont ? 0 : 1;
    st.status = !finite ? CF_NONFINITE : (norm0 > st.tol ? CF_NOT_CONVERGED : CF_OK);
}

// after a step (finish_step's rules)
__device__ __forceinline__ void persist_step(const SolveArgs &A, const PersistArgs &P, bool first, PersistState &st,
                                             double rr, bool stop)
{
    const int k = st.k + 1;
    st.k = k;
    if (rr > st.tol_hi && isfinite(rr) && k < P.max_steps && !stop && P.hist_cap == 0) return;   // goes on
    const double norm = sqrt(rr);
    st.norm = norm;
    persist_record(A, P, first, k, norm);
    const bool finite = isfinite(norm);
    bool cont = finite && k < P.max_steps && (norm > st.tol || k < P.min_steps);
    st.status = !finite ? CF_NONFINITE : (norm > st.tol ? CF_NOT_CONVERGED : CF_OK);
    if (stop) {
        cont = false;
        st.status = CF_TIMEOUT;
    }
    st.done = cont ? 0 : 1;
}

template <int FMT> struct PersistCols;
template <> struct PersistCols<kSell> {
    static __device__ __forceinline__ SellCols32 make(const SolveArgs &A) { return SellCols32{A.s_col}; }
};
template <> struct PersistCols<kSellC> {
    static __device__ __forceinline__ SellCodes8 make(const SolveArgs &A) { return SellCodes8(A.s_code, A.s_dtab); }
};
template <> struct PersistCols<kSellD> {
    static __device__ __forceinline__ SellDelta16 make(const SolveArgs &A) { return SellDelta16{A.s_d16}; }
};

// LOCALM: this block's slots of the matrix and its vectors stay in shared
// memory for the whole solve, and only the gathered vector crosses blocks.
// SYNC: the grid, or one cluster.
template <int SOLVER, int FMT, bool LOCALM, class SYNC>
__global__ void __launch_bounds__(SYNC::kThreads, 1)
    k_persist(const __grid_constant__ SolveArgs A, const __grid_constant__ PersistArgs P)
{
    using Tr = PersistTraits<SOLVER>;
    // in a cluster the gathered vectors live in the blocks' shared memory
    constexpr bool DSM = SYNC::kCluster;
    // Where the matrix streams, the FP64 unit bounds the passes (figures at
    // FixedDot); with a row or two per thread, in shared memory, barriers do and
    // FMA chains are the shorter code (MRJacobi step at 47k rows 8.4 us against
    // 8.7).  CG and PCG keep them at all sizes: their counts over thousands of
    // steps move with the rounding of the sums.
    using Dot = std::conditional_t<LOCALM, PlainDot, FixedDot>;
    const int head = P.head;
    __shared__ typename SYNC::Shared sh;
    __shared__ PersistState st;
    extern __shared__ __align__(16) double local_[];
    if (threadIdx.x == 0) {
        st = PersistState{};
        st.k = -1;   // (no residual yet)
    }
    SYNC gs(P.g, &sh);

    const int n = A.n, ns = A.n_slices;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int rank = gs.rank();
    const bool first_block = rank == 0;
    const bool table = !LOCALM && P.first;
    const int s_lo = table ? P.first[rank] : (int)((int64_t)ns * rank / gs.blocks());
    const int s_hi = table ? P.first[rank + 1] : (int)((int64_t)ns * (rank + 1) / gs.blocks());
    const int base = 32 * s_lo;              // first row of this block
    const uint64_t pol = P.keep ? l2_evict_normal_policy() : l2_evict_first_policy();
    const auto cols = PersistCols<FMT>::make(A);
    const bool has_long = A.has_long != 0;
    double *const xg = A.x;
    const double *b = A.b;
    const double *scale_g = Tr::kScale ? (SOLVER == CF_JMR ? A.corr_scale : A.dinv) : nullptr;
    // block-private vectors, indexed by row - base
    double *q, *rl, *x, *own, *own2 = nullptr;
    const double *scale;
    const int32_t *off;                      // slice offsets, indexed by s - s_lo
    if constexpr (LOCALM) {
        q = local_ + P.plan.q;
        rl = local_ + P.plan.r;
        x = Tr::kLocalX || DSM ? local_ + P.plan.x : xg + base;
        own = local_ + P.plan.g;
        own2 = local_ + P.plan.g2;
        scale = local_ + P.plan.scale;
        off = reinterpret_cast<const int32_t *>(local_ + P.plan.off);
    } else {
        q = P.plan.q >= 0 ? local_ + P.plan.q : (Tr::kMr ? A.w[0] : A.q) + base;
        rl = P.plan.r >= 0 ? local_ + P.plan.r : A.r[0] + base;
        x = P.plan.x >= 0 ? local_ + P.plan.x : xg + base;
        own = (SOLVER == CF_MRJACOBI ? A.w[1] : A.p[0]) + base;
        scale = Tr::kScale ? scale_g + base : nullptr;
        off = P.plan.off >= 0 ? reinterpret_cast<const int32_t *>(local_ + P.plan.off) : A.s_off + s_lo;
    }
    const bool x_local = x != xg + base;
    // r also goes to global memory where the product gathers it
    double *const rg = !DSM && Tr::kGatherR && rl != A.r[0] + base ? A.r[0] + base : nullptr;
    const double *lval = nullptr;
    const int32_t *lcol = nullptr;
    if (LOCALM || P.plan.off >= 0) {
        int32_t *o = reinterpret_cast<int32_t *>(local_ + P.plan.off);
        for (int s = threadIdx.x; s <= s_hi - s_lo; s += blockDim.x) o[s] = A.s_off[s_lo + s];
    }
    if constexpr (LOCALM) {
        const int e0 = A.s_off[s_lo], e1 = A.s_off[s_hi];
        const double *src = Tr::kScaledMatrix ? A.sc_val : A.s_val;
        double *dv = local_ + P.plan.val;
        int32_t *dc = reinterpret_cast<int32_t *>(local_ + P.plan.col);
        for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
            dv[e - e0] = __ldg(src + e);
            const int c = __ldg(A.s_col + e);
            if constexpr (DSM) {
                // the cluster address of row c's element of rl, in the block
                // that owns its slice
                const int t = c >> 5, nb = gs.blocks();
                int o = (int)((int64_t)t * nb / ns);
                while ((int)((int64_t)ns * (o + 1) / nb) <= t) ++o;
                const int o_lo = (int)((int64_t)ns * o / nb);
                dc[e - e0] = (int)(gs.remote(rl, (uint32_t)o) + 8u * (uint32_t)(c - 32 * o_lo));
            } else {
                dc[e - e0] = c;
            }
        }
        for (int i = threadIdx.x; i < 32 * (s_hi - s_lo); i += blockDim.x)
            if (Tr::kScale && base + i < n) local_[P.plan.scale + i] = scale_g[base + i];
        lval = dv;
        lcol = dc;
    }
    __syncthreads();

    // what the product gathers: own rows `mine` of a vector in a cluster (the
    // slots hold the cluster addresses of rl's elements; every vector is at the
    // same place in every block), else the vector itself
    auto gather = [&](const double *mine, const double *global) {
        if constexpr (DSM) {
            const int shift = (int)(reinterpret_cast<const char *>(mine) - reinterpret_cast<const char *>(rl));
            return [shift](int a) {
                double v;
                asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a + shift));
                return v;
            };
        } else {
            return [global](int c) { return global[c]; };
        }
    };
    // this lane's row of slice s over the loop's matrix
    auto product = [&](const double *val, int s, auto g) {
        const int o = off[s - s_lo], len = (off[s - s_lo + 1] - o) >> 5;
        if constexpr (LOCALM) {
            const int l = o - off[0] + lane;
            return local_slice<double, kSellBatch>(lcol + l, lval + l, len, g);
        } else {
            return sell_slice_at<double, kSellBatch>(n, s, o, len, cols, val, A.ro, has_long, pol, g);
        }
    };
    // over A itself (the set-up's products)
    auto product_a = [&](int s, auto g) {
        const int o = off[s - s_lo], len = (off[s - s_lo + 1] - o) >> 5;
        if constexpr (LOCALM && !Tr::kScaledMatrix) {
            const int l = o - off[0] + lane;
            return local_slice<double, kSellBatch>(lcol + l, lval + l, len, g);
        } else {
            return sell_slice_at<double, kSellBatch>(n, s, o, len, cols, A.s_val, A.ro, has_long, pol, g);
        }
    };

    // ---- normFactor and the initial residual -----------------------------
    {
        double acc[1] = {0.0};
        for (int s = s_lo + warp; s < s_hi; s += nw) {
            const int row = 32 * s + lane;
            if (row < n) {
                const double xi = xg[row];
                if (x_local) x[row - base] = xi;
                acc[0] += xi;
            }
        }
        if (!gs.sum(acc, nullptr, [&](const double(&t)[1]) { st.xbar = t[0] / n; })) goto out;
    }
    {
        const double xbar = st.xbar;
        const double cval = P.l1 ? 1.0 : xbar;
        // |A x - A xbar|, |b - A xbar| (squared sums or L1), (r, r), and PCG's (r, D^-1 r)
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        for (int s = s_lo + warp; s < s_hi; s += nw) {
            const int row = 32 * s + lane, i = row - base;
            double y;
            if constexpr (LOCALM && !Tr::kScaledMatrix) y = product_a(s, gather(x, xg));
            else y = product_a(s, [&](int c) { return xg[c]; });
            double yb = product_a(s, [&](int) { return cval; });
            if (P.l1) yb = __dmul_rn(yb, xbar);
            if (row < n) {
                const double bi = b[row];
                const double d1 = y - yb, d2 = bi - yb;
                double ri = bi - y;
                if (SOLVER == CF_JMR) ri = __dmul_rn(A.dinv_sqrt[row], ri);
                rl[i] = ri;
                if (rg) rg[i] = ri;
                if (P.l1) {
                    acc[0] += fabs(d1) + fabs(d2);
                } else {
                    acc[0] = fma_t(d1, d1, acc[0]);
                    acc[1] = fma_t(d2, d2, acc[1]);
                }
                acc[2] = fma_t(ri, ri, acc[2]);
                if (SOLVER == CF_PCG) acc[3] = fma_t(ri, __dmul_rn(scale[i], ri), acc[3]);
                if (SOLVER == CF_MRJACOBI) {
                    const double zi = __dmul_rn(scale[i], ri);
                    if (!DSM) A.w[1][row] = zi;
                    if (LOCALM) own[i] = zi;
                }
            }
        }
        if (!gs.sum(acc, nullptr, [&](const double(&t)[4]) {
                const double nf = P.l1 ? t[0] + 1e-20 : sqrt(t[0]) + sqrt(t[1]) + 1e-20;
                st.nf = nf;
                st.tol = P.abs_tol ? P.tolerance : P.tolerance * nf;
                st.omega = P.omega;
                st.lambda = 0.0;
                persist_begin(A, P, first_block, st, t[2]);
                if (SOLVER == CF_PCG) st.rho0 = t[3];
            }))
            goto out;
    }

    // ---- Richardson's relaxation factor (OptimizePower) -------------------
    if (SOLVER == CF_RICHARDSON && -1e-15 < P.omega && P.omega < 1e-15) {
        const double inv_n = 1.0 / n;
        for (int j = 0; j <= P.power_steps; ++j) {
            // step j: y = A (y_{j-1} / ||y_{j-1}||); the last product gives (v, A v)
            const bool last = j == P.power_steps;
            const double sc = st.pow_inv;
            const double *yp = A.w[(j + 1) & 1];
            double *yn = A.w[j & 1] + base;
            const double *ypl = yp + base;
            if constexpr (DSM) {
                ypl = j & 1 ? own : own2;
                yn = j & 1 ? own2 : own;
            }
            auto gy = gather(ypl, yp);
            auto scaled = [&](double v) { return j == 0 ? inv_n : __dmul_rn(sc, v); };
            double acc[1] = {0.0};
            for (int s = s_lo + warp; s < s_hi; s += nw) {
                const int row = 32 * s + lane, i = row - base;
                double v;
                if (j == 0) v = product_a(s, [&](int) { return inv_n; });
                else v = product_a(s, [&](int c) { return __dmul_rn(sc, gy(c)); });
                if (row < n) {
                    if (!last) yn[i] = v;
                    acc[0] = fma_t(last ? scaled(j == 0 ? 0.0 : ypl[i]) : v, v, acc[0]);
                }
            }
            if (!gs.sum(acc, nullptr, [&](const double(&t)[1]) {
                    if (last) {
                        st.lambda = t[0];
                        st.omega = 2.0 / (t[0] + P.diag_abs_min);
                    } else {
                        st.pow_inv = 1 / sqrt(t[0]);
                    }
                }))
                goto out;
        }
    }

    // ---- the iterations ---------------------------------------------------
    // (element-wise passes take two rows, slices s and s + nw, per round: all
    // loads first)
    for (int k = 1; !st.done; ++k) {
        if constexpr (Tr::kCgLike) {
            double *p = A.p[0];
            {
                const double beta = st.beta, xi = st.xi;
                for (int s = s_lo + warp; s < s_hi; s += 2 * nw) {
                    double pv[2], xv[2], rv[2];
                    bool ok[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int row = 32 * (s + h * nw) + lane, i = row - base;
                        ok[h] = s + h * nw < s_hi && row < n;
                        if (ok[h]) {
                            // PCG: z = D^-1 r, left in q's place by the update (q is dead
                            // there): an FP64 operation of 15 and a load per row fewer, us per
                            // step 14.95 -> 14.55 at 219k rows, 24.4 -> 23.2 at 517k, 68.5 ->
                            // 64.4 at 2.1M
                            if (SOLVER == CF_PCG) rv[h] = k > 1 ? q[i] : __dmul_rn(scale[i], rl[i]);
                            else rv[h] = rl[i];
                            if (k > 1) {
                                pv[h] = own[i];
                                xv[h] = x[i];
                            }
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (ok[h]) {
                            const int row = 32 * (s + h * nw) + lane, i = row - base;
                            if (k > 1) {
                                x[i] = fma_t(xi, pv[h], xv[h]);
                                rv[h] = fma_t(beta, pv[h], rv[h]);
                            }
                            if (!DSM) p[row] = rv[h];
                            if (LOCALM) own[i] = rv[h];
                        }
                }
            }
            if (!gs.barrier()) goto out;
            {
                // the reciprocal the next beta needs, off the critical path
                if (threadIdx.x == blockDim.x - 32) st.rrho = 1.0 / st.rho0;
                double acc[1] = {0.0};
                for (int s = s_lo + warp; s < s_hi; s += nw) {
                    const int row = 32 * s + lane;
                    const double y = product(A.s_val, s, gather(own, p));
                    if (row < n) {
                        q[row - base] = y;
                        acc[0] = fma_t(own[row - base], y, acc[0]);
                    }
                }
                if (!gs.sum(acc, nullptr, [&](const double(&t)[1]) { st.xi = st.rho0 / t[0]; })) goto out;
            }
            {
                const double xi = st.xi;
                double acc[2] = {0.0, 0.0};
                for (int s = s_lo + warp; s < s_hi; s += 2 * nw) {
                    double qv[2], rv[2];
                    bool ok[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int row = 32 * (s + h * nw) + lane, i = row - base;
                        ok[h] = s + h * nw < s_hi && row < n;
                        if (ok[h]) {
                            qv[h] = q[i];
                            rv[h] = rl[i];
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (ok[h]) {
                            const int i = 32 * (s + h * nw) + lane - base;
                            const double ri = fma_t(-xi, qv[h], rv[h]);
                            rl[i] = ri;
                            acc[0] = fma_t(ri, ri, acc[0]);
                            if (SOLVER == CF_PCG) {
                                const double zi = __dmul_rn(scale[i], ri);
                                q[i] = zi;
                                acc[1] = fma_t(ri, zi, acc[1]);
                            }
                        }
                }
                auto step = [&](double rr, double rho) {
                    st.beta = div_by_reciprocal(rho, st.rho0, st.rrho);
                    st.rho0 = rho;
                    persist_step(A, P, first_block, st, rr, sh.stop != 0);
                };
                bool ok;
                if constexpr (SOLVER == CF_PCG) {
                    ok = gs.sum(acc, A.abort_flag, [&](const double(&t)[2]) { step(t[0], t[1]); });
                } else {
                    const double a1[1] = {acc[0]};
                    ok = gs.sum(a1, A.abort_flag, [&](const double(&t)[1]) { step(t[0], t[0]); });
                }
                if (!ok) goto out;
            }
        } else if constexpr (Tr::kMr) {
            // y = A r (A z, or L A R r), (r, y), (y, y)
            double *gv = SOLVER == CF_MRJACOBI ? A.w[1] : A.r[0];
            {
                const double *val = Tr::kScaledMatrix ? A.sc_val : A.s_val;
                Dot acc[2];
                for (int s = s_lo + warp; s < s_hi; s += nw) {
                    const int row = 32 * s + lane, i = row - base;
                    const double y = product(val, s, gather(SOLVER == CF_MRJACOBI ? own : rl, gv));
                    if (row < n) {
                        q[i] = y;
                        acc[0].add(rl[i], y, head);
                        acc[1].add(y, y, head);
                    }
                }
                if (!gs.sum(acc, nullptr, [&](const double(&t)[2]) { st.omega = t[0] / t[1]; }, head)) goto out;
            }
            const double alpha = st.omega;
            Dot acc[1];
            for (int s = s_lo + warp; s < s_hi; s += 2 * nw) {
                double rv[2], xv[2], yv[2], dv[2], sv[2];
                bool ok[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int row = 32 * (s + h * nw) + lane, i = row - base;
                    ok[h] = s + h * nw < s_hi && row < n;
                    if (ok[h]) {
                        rv[h] = rl[i];
                        xv[h] = x[i];
                        yv[h] = q[i];
                        if (SOLVER == CF_MRJACOBI) {
                            dv[h] = own[i];
                            sv[h] = scale[i];
                        } else {
                            dv[h] = SOLVER == CF_JMR ? __dmul_rn(scale[i], rv[h]) : rv[h];
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (ok[h]) {
                        const int row = 32 * (s + h * nw) + lane, i = row - base;
                        x[i] = fma_t(alpha, dv[h], xv[h]);
                        const double ri = fma_t(-alpha, yv[h], rv[h]);
                        rl[i] = ri;
                        if (rg) rg[i] = ri;
                        if (SOLVER == CF_MRJACOBI) {
                            const double zi = __dmul_rn(sv[h], ri);
                            if (!DSM) gv[row] = zi;
                            if (LOCALM) own[i] = zi;
                        }
                        acc[0].add(ri, ri, head);
                    }
            }
            if (!gs.sum(acc, A.abort_flag,
                        [&](const double(&t)[1]) { persist_step(A, P, first_block, st, t[0], sh.stop != 0); }, head))
                goto out;
        } else if constexpr (SOLVER == CF_JACOBI) {
            // one pass over A D^-1: the residual alternates between r[0] and r[1]
            const double *rin = A.r[(k + 1) & 1];
            double *rout = A.r[k & 1] + base;
            const double *mine = rin + base;
            if constexpr (DSM) {
                mine = k & 1 ? rl : own2;
                rout = k & 1 ? own2 : rl;
            } else if constexpr (LOCALM) {
                mine = rl;
            }
            Dot acc[1];
            for (int s = s_lo + warp; s < s_hi; s += nw) {
                const int row = 32 * s + lane, i = row - base;
                const double y = product(A.sc_val, s, gather(mine, rin));
                if (row < n) {
                    const double r0 = mine[i];
                    x[i] = fma_t(1.0, __dmul_rn(scale[i], r0), x[i]);
                    const double ri = fma_t(-1.0, y, r0);
                    rout[i] = ri;
                    if (LOCALM && !DSM) rl[i] = ri;
                    acc[0].add(ri, ri, head);
                }
            }
            if (!gs.sum(acc, A.abort_flag,
                        [&](const double(&t)[1]) { persist_step(A, P, first_block, st, t[0], sh.stop != 0); }, head))
                goto out;
        } else {
            // Richardson: x += omega r; r = b - A x
            const double omega = st.omega;
            for (int s = s_lo + warp; s < s_hi; s += nw) {
                const int row = 32 * s + lane;
                if (row < n) x[row - base] = fma_t(omega, rl[row - base], x[row - base]);
            }
            if (!gs.barrier()) goto out;
            Dot acc[1];
            for (int s = s_lo + warp; s < s_hi; s += nw) {
                const int row = 32 * s + lane;
                const double t = product(A.s_val, s, gather(x, xg));
                if (row < n) {
                    const double ri = b[row] - t;
                    rl[row - base] = ri;
                    acc[0].add(ri, ri, head);
                }
            }
            if (!gs.sum(acc, A.abort_flag,
                        [&](const double(&t)[1]) { persist_step(A, P, first_block, st, t[0], sh.stop != 0); }, head))
                goto out;
        }
    }
    // x back, with the last step of CG
    if (x_local || Tr::kCgLike) {
        const double xi = st.xi;
        const bool last = Tr::kCgLike && st.k > 0;
        for (int s = s_lo + warp; s < s_hi; s += nw) {
            const int row = 32 * s + lane, i = row - base;
            if (row < n) xg[row] = last ? fma_t(xi, own[i], x[i]) : x[i];
        }
    }
out:
    if (first_block && threadIdx.x == 0) {
        DevState *o = P.out;
        o->nf = st.nf;
        o->norm0 = st.norm0;
        o->norm = st.norm;
        o->omega = st.omega;
        o->lambda_max = st.lambda;
        o->k = st.k;
        o->status = st.status;
    }
    report_fail(sh.fail, P.out);
    gs.leave();
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
template <int SOLVER>
static const void *persist_pick(int scope, int format)
{
    if (scope == kScopeCluster) return (const void *)k_persist<SOLVER, kSell, true, ClusterSync>;
    if (scope == kScopeGridLocal) return (const void *)k_persist<SOLVER, kSell, true, GridSync>;
    return format == kSellC   ? (const void *)k_persist<SOLVER, kSellC, false, GridSync>
           : format == kSellD ? (const void *)k_persist<SOLVER, kSellD, false, GridSync>
                              : (const void *)k_persist<SOLVER, kSell, false, GridSync>;
}

// the vectors a solver keeps per block
struct PersistNeeds {
    bool q, gather_r, own, local_x, scale;
};
template <int SOLVER> static PersistNeeds needs_of()
{
    using Tr = PersistTraits<SOLVER>;
    return {Tr::kQ, Tr::kGatherR, Tr::kOwnG, Tr::kLocalX, Tr::kScale};
}
static PersistNeeds persist_needs(int solver)
{
    switch (solver) {
    case CF_CG: return needs_of<CF_CG>();
    case CF_PCG: return needs_of<CF_PCG>();
    case CF_JACOBI: return needs_of<CF_JACOBI>();
    case CF_RICHARDSON: return needs_of<CF_RICHARDSON>();
    case CF_MR: return needs_of<CF_MR>();
    case CF_JMR: return needs_of<CF_JMR>();
    default: return needs_of<CF_MRJACOBI>();   // (MRS too)
    }
}

static const void *persist_kernel(int solver, int scope, int format)
{
    switch (solver) {
    case CF_CG: return persist_pick<CF_CG>(scope, format);
    case CF_PCG: return persist_pick<CF_PCG>(scope, format);
    case CF_JACOBI: return persist_pick<CF_JACOBI>(scope, format);
    case CF_RICHARDSON: return persist_pick<CF_RICHARDSON>(scope, format);
    case CF_MR: return persist_pick<CF_MR>(scope, format);
    case CF_MRJACOBI:
    case CF_MRS: return persist_pick<CF_MRJACOBI>(scope, format);
    case CF_JMR: return persist_pick<CF_JMR>(scope, format);
    default: return nullptr;
    }
}

// Cooperative launches, and no more SMs than the partial sums are sized for.
bool persist_possible(Context *ctx)
{
    if (ctx->sm_count > kPMaxGrid) return false;
    if (ctx->coop_ok < 0) {
        int coop = 0;
        if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device) != cudaSuccess) {
            cudaGetLastError();
            coop = 0;
        }
        ctx->coop_ok = coop;
    }
    return ctx->coop_ok == 1;
}

// Whether a solve over the SELL-32 copy runs here.  CSR matrices (their staging
// buffers), BiCG's fast order and devices where it is not possible run the
// multi-kernel loop, and so do large systems:
//
// * FP64.  A block's rows are contiguous, so at any time 152 windows of the
//   gathered vector are in use, each twice the largest column offset; the loop
//   deals slices round robin and has one.  Once the windows (at most the whole
//   vector) outgrow their part of L2 the loop is faster.  us per step, here /
//   loop: CG 176^3 153 / 159, 208^3 254 / 254, 224^3 323 / 311, 256^3 473 / 450;
//   MR 208^3 212 / 213, 256^3 400 / 379; PCG 208^3 293 / 293, 256^3 540 / 524;
//   Jacobi 192^3 151 / 155, 208^3 200 / 195; MRJacobi, which gathers z beside r,
//   176^3 169 / 170, 192^3 218 / 214, 256^3 515 / 479.  Narrow windows stay here:
//   4096^2 CG 397 / 419, MRJacobi 436 / 449; 64 x 64 x 4096 CG 436 / 450.
// * Richardson, one product per step: 176^3 128 / 129, 192^3 168 / 164, 256^3 411
//   / 369; 4096^2 351 / 340.
// * FP32 sweeps: past L2 their products are bound by loads in flight, 32 warps
//   per SM here and 48 in the loop.  MR 160^3 46 / 49, 176^3 61 / 61, 256^3 225 /
//   199; MRJacobi, JMR 176^3 71 / 75, 192^3 99 / 97, 256^3 254 / 231; BiCGStab 208^3
//   312 / 317, 224^3 388 / 387, 256^3 598 / 558; CG is faster here at every size
//   (288^3 399 / 445).
//
// The limits are shares of L2 (135.5 MB) that 8 bytes per row, or the windows,
// take: 0.53 is 9M rows.
bool persist_usable(Context *ctx, int solver, int format, bool mixed, const Matrix *m)
{
    if (format == kCsr || !persist_possible(ctx)) return false;
    if (!mixed && !persist_kernel(solver, kScopeGrid, format)) return false;
    const double l2 = (double)ctx->l2_bytes;
    const double vector = 8.0 * m->n, windows = std::min(vector, 16.0 * m->max_offset * ctx->sm_count);
    const bool diag = solver == CF_MRJACOBI || solver == CF_MRS;
    if (mixed)
        return solver == CF_CG || vector <= (solver == CF_BICG ? 0.65 : diag || solver == CF_JMR ? 0.385 : 0.32) * l2;
    if (solver == CF_RICHARDSON) return vector <= 0.355 * l2;
    return windows <= (diag ? 0.325 : solver == CF_JACOBI ? 0.47 : 0.53) * l2;
}

// Asked for the kernel to be launched, with its own registers and the most
// dynamic shared memory it is given, once per context: where the answer is no,
// its solves run on the grid.
bool persist_cluster_fits(Context *ctx, const void *kernel)
{
    const auto seen = ctx->cluster_fits.find(kernel);
    if (seen != ctx->cluster_fits.end()) return seen->second;
    raise_smem_limit(kernel, persist_smem_limit(true));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kPClusterMax;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(ClusterSync::kThreads);
    cfg.gridDim = dim3(kPClusterMax);
    cfg.dynamicSmemBytes = persist_smem_limit(true);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters >= 1;
    cudaGetLastError();
    return ctx->cluster_fits[kernel] = ok;
}

PersistGrid persist_grid(Context *ctx)
{
    const size_t part = sizeof(double) * 2 * kPMaxNV * kPMaxGrid;
    if (ctx->persist.bytes == 0) {
        ctx->persist.ensure(part + 64);
        CF_CUDA(cudaMemsetAsync(ctx->persist.ptr, 0, part + 64, ctx->stream));
    }
    PersistGrid g;
    g.part = ctx->persist.as<double>();
    g.count = reinterpret_cast<uint32_t *>(static_cast<char *>(ctx->persist.ptr) + part);
    g.stop = reinterpret_cast<int32_t *>(g.count + 4);
    g.poll_limit = ctx->poll_limit;
    return g;
}

void launch_persist_kernel(Context *ctx, const void *kernel, bool cluster, int grid, int slices_per_block,
                           size_t smem, void **args)
{
    raise_smem_limit(kernel, persist_smem_limit(cluster));
    const int warps = std::max(4, std::min(kPWarps, (slices_per_block + 3) / 4 * 4));
    if (!cluster) {
        CF_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(32 * warps), args, smem, ctx->stream));
        return;
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = grid;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(32 * warps);
    cfg.gridDim = dim3(grid);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (grid > 8) CF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    CF_CUDA(cudaLaunchKernelExC(&cfg, kernel, args));
}

// Equal numbers of slices are unequal work where the rows of one part of the
// numbering are longer (a refined or polyhedral region): every pass waits for the
// blocks of the long part.  There the blocks are dealt equal costs, a slice's
// slots per row plus kShareVector for the vector passes (a CG step has 12 FP64
// operations per 7-point row, five of them outside the product).  Measured on
// GB300, us per 60 steps, the last tenth of the rows 15 long and the others 7,
// equal numbers -> equal costs, CG / Jacobi / mixed CG: 0.5M rows 1,639 -> 1,393 /
// 1,229 -> 931 / 1,035 -> 923; 2M rows 4,907 -> 3,903 / 4,119 -> 2,855 / 2,891 ->
// 2,303 (the multi-kernel loop, which deals slices round robin: 4,623 / 3,562 /
// 3,457).
constexpr int kShareVector = 5;
// ... where the longest slice costs this much more than the mean one
constexpr double kShareUneven = 1.05;

// first[0 .. grid]: the blocks' first slices, at equal steps of the running cost;
// returns the most slices of a block
static int share_slices(const int32_t *off, int ns, int grid, int32_t *first)
{
    auto cost = [&](int s) { return (int64_t)off[s] / 32 + (int64_t)kShareVector * s; };
    const int64_t total = cost(ns);
    int s = 0, most = 0;
    first[0] = 0;
    for (int b = 1; b <= grid; ++b) {
        const int64_t want = total * b / grid;
        while (s < ns && cost(s) < want) ++s;
        first[b] = b == grid ? ns : s;
        most = std::max(most, first[b] - first[b - 1]);
    }
    return most;
}

const int32_t *persist_shares(Matrix *m, int grid, int &most)
{
    const int ns = m->n_slices;
    most = (ns + grid - 1) / grid;
    if (m->sell_max_len + kShareVector <= kShareUneven * ((double)m->sell_nnz / (32.0 * ns) + kShareVector))
        return nullptr;
    if (m->share_blocks != grid) {   // (once per pattern)
        std::vector<int32_t> off((size_t)ns + 1), first((size_t)grid + 1);
        m->share_blocks = 0;
        CF_CUDA(cudaMemcpyAsync(off.data(), m->s_off.ptr, sizeof(int32_t) * off.size(), cudaMemcpyDeviceToHost,
                                m->ctx->stream));
        CF_CUDA(cudaStreamSynchronize(m->ctx->stream));
        m->share_most = share_slices(off.data(), ns, grid, first.data());
        m->shares.ensure(sizeof(int32_t) * first.size());
        // (a pageable source: staged when the call returns)
        CF_CUDA(cudaMemcpyAsync(m->shares.ptr, first.data(), sizeof(int32_t) * first.size(), cudaMemcpyHostToDevice,
                                m->ctx->stream));
        m->share_blocks = grid;
    }
    most = m->share_most;
    return m->shares.as<int32_t>();
}

void launch_persist(Context *ctx, int solver, int format, const SolveArgs &A, const DevState &S, int l1, Matrix *m,
                    DevState *out)
{
    const int max_len = m->sell_max_len;   // slots per row of the longest slice
    PersistArgs P;
    std::memset(&P, 0, sizeof(P));
    P.g = persist_grid(ctx);
    P.out = out;
    P.tolerance = S.tolerance;
    P.rel_tol = S.rel_tol;
    P.omega = S.omega;
    P.diag_abs_min = S.diag_abs_min;
    P.max_steps = S.max_steps;
    P.min_steps = S.min_steps;
    P.hist_cap = S.hist_cap;
    P.abs_tol = (S.flags & kFlagAbsTol) ? 1 : 0;
    P.l1 = l1;
    P.power_steps = A.power_steps;

    const PersistNeeds need = persist_needs(solver);
    const int ns = A.n_slices;
    // everything a block of `slices` slices keeps in shared memory, in doubles
    auto plan_all = [&](int slices, bool cluster) {
        PersistPlan p;
        int at = 0;
        auto take = [&](int doubles) {
            const int o = at;
            at += doubles;
            return o;
        };
        p.off = take(slices / 2 + 2);
        p.q = need.q ? take(32 * slices) : -1;
        p.r = take(32 * slices);
        p.x = need.local_x || cluster ? take(32 * slices) : -1;
        p.scale = need.scale ? take(32 * slices) : -1;
        const bool power = cluster && solver == CF_RICHARDSON;
        p.g = need.own || power ? take(32 * slices) : -1;
        p.g2 = power || (cluster && solver == CF_JACOBI) ? take(32 * slices) : -1;
        p.val = take(32 * slices * max_len);
        p.col = take(16 * slices * max_len);
        return std::make_pair(p, sizeof(double) * (size_t)at);
    };

    int scope = kScopeGrid, grid = 1, most = 0;   // (most: slices of a block)
    size_t smem = 0;
    if (A.n <= CF_PERSIST_CLUSTER_ROWS && !A.has_long &&
        persist_cluster_fits(ctx, persist_kernel(solver, kScopeCluster, format))) {
        // one warp per sub-partition and block before another block is added
        grid = 1;
        while (grid < 16 && 4 * grid < ns) grid <<= 1;
        const auto pl = plan_all((ns + grid - 1) / grid, true);
        if (pl.second + sizeof(ClusterSync::Shared) <= CF_PERSIST_LOCAL_BYTES) {
            scope = kScopeCluster;
            P.plan = pl.first;
            smem = pl.second;
        }
    }
    if (scope == kScopeGrid) {
        grid = std::max(1, std::min(ctx->sm_count, (ns + 3) / 4));
        const int slices = (ns + grid - 1) / grid;
        const auto pl = slices <= 4096 && max_len <= 64 ? plan_all(slices, false) : std::make_pair(PersistPlan{}, ~(size_t)0);
        if (!A.has_long && pl.second <= CF_PERSIST_LOCAL_BYTES) {
            scope = kScopeGridLocal;
            P.plan = pl.first;
            smem = pl.second;
        } else {
            // vectors only, as many as fit: q and r first, then x
            P.first = persist_shares(m, grid, most);
            int at = 0;
            const int cap = CF_PERSIST_VEC_BYTES / (int)sizeof(double);
            auto take = [&](bool want, int doubles) {
                if (!want || at + doubles > cap) return -1;
                const int o = at;
                at += doubles;
                return o;
            };
            P.plan.val = P.plan.col = P.plan.scale = P.plan.g = P.plan.g2 = -1;
            P.plan.off = take(most <= 4096, most / 2 + 2);
            P.plan.q = take(most <= 4096 && need.q, 32 * most);
            P.plan.r = take(most <= 4096 && !need.gather_r, 32 * most);
            P.plan.x = take(most <= 4096 && need.local_x, 32 * most);
            smem = sizeof(double) * (size_t)at;
        }
    }
    // 893k rows (75 MB of slots, 36 MB of vectors): CG step 29.1 us with the
    // evict-first hint, 27.0 without; 2.1M rows (176 MB) need it
    const double slots = 12.0 * (double)m->sell_nnz, vectors = 40.0 * A.n;
    P.keep = slots + vectors < 0.95 * (double)ctx->l2_bytes ? 1 : 0;
    const void *kernel = persist_kernel(solver, scope, format);
    if (!most) most = (ns + grid - 1) / grid;
    const int slices_per_warp = (most + kPWarps - 1) / kPWarps;
    P.head = 2;
    while ((1 << (P.head - 1)) <= slices_per_warp) ++P.head;
    SolveArgs a = A;
    void *args[] = {&a, &P};
    out->flags = 0;   // (S may be *out: read above)
    launch_persist_kernel(ctx, kernel, scope == kScopeCluster, grid, most, smem, args);
}

// after a solve whose blocks gave up waiting: the arrival counter is not zero
void persist_reset(Context *ctx) { ctx->persist.release(); }

} // namespace cf
