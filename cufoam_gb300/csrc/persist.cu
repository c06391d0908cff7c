// persist.cu -- FP64 solves in the fast summation order as one cooperative
// launch: normFactor, the initial residual, every step and the last update
// of psi, with a grid barrier where the multi-kernel loop (solve_fast.cu)
// has a kernel boundary.
//
// What bounds the multi-kernel loop below about a million rows is not bytes
// or FP64 issue but its boundaries: launch, ramp-up, drain and the last
// block's serial reduction, 4 to 8 us per kernel.  A grid barrier costs 1.2
// us here, a grid sum about 2.5.  Measured on GB300, us per step and for
// normFactor + residual + first step (7-point systems, multi-kernel loop ->
// here):
//                 22k rows     219k rows    893k rows    2.1M rows
//   CG step       16.6->10.7   28.8->14.2   43.9->29.6   72.1->59.6
//   Jacobi step    8.3-> 4.7   15.3-> 8.6   28.8->22.2   53.5->46.4
//   MR step       15.2->11.3   23.8->13.8   37.8->28.6   62.9->54.7
//   CG set-up     102 -> 39    160 -> 49    267 -> 92    422 -> 178
// The arithmetic of a row and of an element
// is the loop's: one FMA chain per row in entry order, one FMA per update;
// only the order of the dot products' partial sums differs.
#include "persist.cuh"

#include <algorithm>
#include <climits>
#include <cstring>

namespace cf {

struct PersistArgs {
    PersistGrid g;
    DevState *out;           // host-mapped: the final state
    double tolerance, rel_tol, omega, diag_abs_min;
    int32_t max_steps, min_steps, hist_cap;
    int32_t abs_tol, l1, power_steps;
    int32_t local_rows;      // rows per block of the block-private vectors in shared memory (0: in global)
};

// Per-block step state, the same bits in every block (thread 0 writes it
// between barriers).
struct PersistState {
    double rho0, rho1, xi, beta, omega, tol, nf, norm, norm0, xbar, pow_inv, lambda;
    int32_t k, done, status;
};

// CF_CG, CF_PCG, CF_JACOBI, CF_RICHARDSON, CF_MR; MRJacobi and MRS run as
// CF_MRJACOBI (z = D^-1 r gathered), JMR as CF_JMR (MR on the scaled matrix)
template <int SOLVER> struct PersistTraits {
    static constexpr bool kCgLike = SOLVER == CF_CG || SOLVER == CF_PCG;
    static constexpr bool kMr = SOLVER == CF_MR || SOLVER == CF_MRJACOBI || SOLVER == CF_JMR;
    // r read by other blocks (gathered by the product)
    static constexpr bool kGatherR = SOLVER == CF_MR || SOLVER == CF_JMR || SOLVER == CF_JACOBI;
};

__device__ __forceinline__ void persist_record(const SolveArgs &A, const PersistArgs &P, int k, double norm)
{
    if (blockIdx.x == 0 && k < P.hist_cap) {
        if (A.hist) A.hist[k] = norm;
        if (A.hist_t) A.hist_t[k] = global_ns();
    }
}

// after the initial residual (finish_init's rules)
__device__ __forceinline__ void persist_begin(const SolveArgs &A, const PersistArgs &P, PersistState &st, double rr)
{
    const double norm0 = sqrt(rr);
    st.rho0 = rr;
    st.rho1 = 0.0;
    st.norm0 = st.norm = norm0;
    persist_record(A, P, 0, norm0);
    if (P.rel_tol > 0.0) st.tol = fmax(st.tol, P.rel_tol * norm0);
    st.k = 0;
    const bool finite = isfinite(norm0);
    const bool cont = finite && P.max_steps >= 1 && (norm0 > st.tol || P.min_steps > 0);
    st.done = cont ? 0 : 1;
    st.status = !finite ? CF_NONFINITE : (norm0 > st.tol ? CF_NOT_CONVERGED : CF_OK);
}

// after a step (finish_step's rules)
__device__ __forceinline__ void persist_step(const SolveArgs &A, const PersistArgs &P, PersistState &st, double rr,
                                             bool stop)
{
    const double norm = sqrt(rr);
    const int k = st.k + 1;
    st.k = k;
    st.norm = norm;
    persist_record(A, P, k, norm);
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

template <int SOLVER, int FMT>
__global__ void __launch_bounds__(kPBlock, 1)
    k_persist(const __grid_constant__ SolveArgs A, const __grid_constant__ PersistArgs P)
{
    using Tr = PersistTraits<SOLVER>;
    __shared__ PersistShared sh;
    __shared__ PersistState st;
    extern __shared__ __align__(16) double local_[];
    PersistSync gs;
    gs.init(P.g, &sh);

    const int n = A.n, ns = A.n_slices;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int s_lo = (int)((int64_t)ns * blockIdx.x / gridDim.x);
    const int s_hi = (int)((int64_t)ns * (blockIdx.x + 1) / gridDim.x);
    const int base = 32 * s_lo;              // first row of this block
    const uint64_t pol = l2_evict_first_policy();
    const auto cols = PersistCols<FMT>::make(A);
    const bool has_long = A.has_long != 0;
    double *x = A.x;
    const double *b = A.b;
    // block-private vectors, indexed by row - base
    double *q = P.local_rows ? local_ : (Tr::kMr ? A.w[0] : A.q) + base;
    double *rl = (P.local_rows && !Tr::kGatherR) ? local_ + (SOLVER == CF_RICHARDSON ? 0 : P.local_rows)
                                                 : A.r[0] + base;

    auto product = [&](const double *val, int s, const double *v) {
        return sell_slice<double, kSellBatch>(n, s, A.s_off, cols, val, A.ro, has_long, pol,
                                              [&](int c) { return v[c]; });
    };

    // ---- normFactor and the initial residual -----------------------------
    {
        double acc[1] = {0.0};
        for (int s = s_lo + warp; s < s_hi; s += kPWarps) {
            const int row = 32 * s + lane;
            if (row < n) acc[0] += x[row];
        }
        if (!gs.sum(acc, nullptr, [&](const double(&t)[1]) { st.xbar = t[0] / n; })) goto out;
    }
    {
        const double xbar = st.xbar;
        const double cval = P.l1 ? 1.0 : xbar;
        // |A x - A xbar|, |b - A xbar| (squared sums or L1), (r, r), and PCG's (r, D^-1 r)
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        for (int s = s_lo + warp; s < s_hi; s += kPWarps) {
            const int row = 32 * s + lane;
            const double y = product(A.s_val, s, x);
            double yb = sell_slice<double, kSellBatch>(n, s, A.s_off, cols, A.s_val, A.ro, has_long, pol,
                                                       [&](int) { return cval; });
            if (P.l1) yb = __dmul_rn(yb, xbar);
            if (row < n) {
                const double bi = b[row];
                const double d1 = y - yb, d2 = bi - yb;
                double ri = bi - y;
                if (SOLVER == CF_JMR) ri = __dmul_rn(A.dinv_sqrt[row], ri);
                rl[row - base] = ri;
                if (P.l1) {
                    acc[0] += fabs(d1) + fabs(d2);
                } else {
                    acc[0] = fma_t(d1, d1, acc[0]);
                    acc[1] = fma_t(d2, d2, acc[1]);
                }
                acc[2] = fma_t(ri, ri, acc[2]);
                if (SOLVER == CF_PCG) acc[3] = fma_t(ri, __dmul_rn(A.dinv[row], ri), acc[3]);
                if (SOLVER == CF_MRJACOBI) A.w[1][row] = __dmul_rn(A.dinv[row], ri);
            }
        }
        if (!gs.sum(acc, nullptr, [&](const double(&t)[4]) {
                const double nf = P.l1 ? t[0] + 1e-20 : sqrt(t[0]) + sqrt(t[1]) + 1e-20;
                st.nf = nf;
                st.tol = P.abs_tol ? P.tolerance : P.tolerance * nf;
                st.omega = P.omega;
                st.lambda = 0.0;
                persist_begin(A, P, st, t[2]);
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
            double *yn = A.w[j & 1];
            double acc[1] = {0.0};
            for (int s = s_lo + warp; s < s_hi; s += kPWarps) {
                const int row = 32 * s + lane;
                auto g = [&](int c) { return j == 0 ? inv_n : __dmul_rn(sc, yp[c]); };
                const double v = sell_slice<double, 4>(n, s, A.s_off, cols, A.s_val, A.ro, has_long, pol, g);
                if (row < n) {
                    if (!last) yn[row] = v;
                    acc[0] = fma_t(last ? g(row) : v, v, acc[0]);
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
    for (int k = 1; !st.done; ++k) {
        if constexpr (Tr::kCgLike) {
            double *p = A.p[0];
            const double *dinv = A.dinv;
            const double beta = st.beta, xi0 = st.xi;
            for (int s = s_lo + warp; s < s_hi; s += 2 * kPWarps) {
                // two rows (slices s and s + 32) per step, all loads first
                double pv[2], xv[2], rv[2];
                bool ok[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int row = 32 * (s + h * kPWarps) + lane;
                    ok[h] = s + h * kPWarps < s_hi && row < n;
                    if (ok[h]) {
                        rv[h] = rl[row - base];
                        if (SOLVER == CF_PCG) rv[h] = __dmul_rn(dinv[row], rv[h]);
                        if (k > 1) {
                            pv[h] = p[row];
                            xv[h] = x[row];
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (ok[h]) {
                        const int row = 32 * (s + h * kPWarps) + lane;
                        if (k > 1) {
                            x[row] = fma_t(xi0, pv[h], xv[h]);
                            p[row] = fma_t(beta, pv[h], rv[h]);
                        } else {
                            p[row] = rv[h];
                        }
                    }
            }
            if (!gs.barrier()) goto out;
            {
                double acc[1] = {0.0};
                for (int s = s_lo + warp; s < s_hi; s += kPWarps) {
                    const int row = 32 * s + lane;
                    const double y = product(A.s_val, s, p);
                    if (row < n) {
                        q[row - base] = y;
                        acc[0] = fma_t(p[row], y, acc[0]);
                    }
                }
                if (!gs.sum(acc, nullptr, [&](const double(&t)[1]) { st.xi = st.rho0 / t[0]; })) goto out;
            }
            {
                const double xi = st.xi;
                double acc[2] = {0.0, 0.0};
                for (int s = s_lo + warp; s < s_hi; s += 2 * kPWarps) {
                    double qv[2], rv[2];
                    bool ok[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int row = 32 * (s + h * kPWarps) + lane;
                        ok[h] = s + h * kPWarps < s_hi && row < n;
                        if (ok[h]) {
                            qv[h] = q[row - base];
                            rv[h] = rl[row - base];
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (ok[h]) {
                            const int row = 32 * (s + h * kPWarps) + lane;
                            const double ri = fma_t(-xi, qv[h], rv[h]);
                            rl[row - base] = ri;
                            acc[0] = fma_t(ri, ri, acc[0]);
                            if (SOLVER == CF_PCG) acc[1] = fma_t(ri, __dmul_rn(dinv[row], ri), acc[1]);
                        }
                }
                bool ok;
                if (SOLVER == CF_PCG) {
                    ok = gs.sum(acc, A.abort_flag, [&](const double(&t)[2]) {
                        st.rho1 = st.rho0;
                        st.rho0 = t[1];
                        st.beta = st.rho0 / st.rho1;
                        persist_step(A, P, st, t[0], sh.stop != 0);
                    });
                } else {
                    const double a1[1] = {acc[0]};
                    ok = gs.sum(a1, A.abort_flag, [&](const double(&t)[1]) {
                        st.rho1 = st.rho0;
                        st.rho0 = t[0];
                        st.beta = st.rho0 / st.rho1;
                        persist_step(A, P, st, t[0], sh.stop != 0);
                    });
                }
                if (!ok) goto out;
            }
        } else if constexpr (Tr::kMr) {
            // y = A r (A z, or L A R r), (r, y), (y, y)
            double *gv = SOLVER == CF_MRJACOBI ? A.w[1] : A.r[0];
            const double *val = SOLVER == CF_JMR ? A.sc_val : A.s_val;
            {
                double acc[2] = {0.0, 0.0};
                for (int s = s_lo + warp; s < s_hi; s += kPWarps) {
                    const int row = 32 * s + lane;
                    const double y = product(val, s, gv);
                    if (row < n) {
                        q[row - base] = y;
                        acc[0] = fma_t(rl[row - base], y, acc[0]);
                        acc[1] = fma_t(y, y, acc[1]);
                    }
                }
                if (!gs.sum(acc, nullptr, [&](const double(&t)[2]) { st.omega = t[0] / t[1]; })) goto out;
            }
            const double alpha = st.omega;
            const double *R = SOLVER == CF_MRJACOBI ? A.dinv : A.corr_scale;
            double acc[1] = {0.0};
            for (int s = s_lo + warp; s < s_hi; s += 2 * kPWarps) {
                double rv[2], xv[2], yv[2], dv[2], sv[2];
                bool ok[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int row = 32 * (s + h * kPWarps) + lane;
                    ok[h] = s + h * kPWarps < s_hi && row < n;
                    if (ok[h]) {
                        rv[h] = rl[row - base];
                        xv[h] = x[row];
                        yv[h] = q[row - base];
                        if (SOLVER == CF_MRJACOBI) {
                            dv[h] = gv[row];
                            sv[h] = R[row];
                        } else {
                            dv[h] = SOLVER == CF_JMR ? __dmul_rn(R[row], rv[h]) : rv[h];
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (ok[h]) {
                        const int row = 32 * (s + h * kPWarps) + lane;
                        x[row] = fma_t(alpha, dv[h], xv[h]);
                        const double ri = fma_t(-alpha, yv[h], rv[h]);
                        rl[row - base] = ri;
                        if (SOLVER == CF_MRJACOBI) gv[row] = __dmul_rn(sv[h], ri);
                        acc[0] = fma_t(ri, ri, acc[0]);
                    }
            }
            if (!gs.sum(acc, A.abort_flag,
                        [&](const double(&t)[1]) { persist_step(A, P, st, t[0], sh.stop != 0); }))
                goto out;
        } else if constexpr (SOLVER == CF_JACOBI) {
            // one pass over A D^-1: the residual alternates between r[0] and r[1]
            const double *rin = A.r[(k + 1) & 1];
            double *rout = A.r[k & 1];
            double acc[1] = {0.0};
            for (int s = s_lo + warp; s < s_hi; s += kPWarps) {
                const int row = 32 * s + lane;
                const double y = product(A.sc_val, s, rin);
                if (row < n) {
                    const double r0 = rin[row];
                    x[row] = fma_t(1.0, __dmul_rn(A.dinv[row], r0), x[row]);
                    const double ri = fma_t(-1.0, y, r0);
                    rout[row] = ri;
                    acc[0] = fma_t(ri, ri, acc[0]);
                }
            }
            if (!gs.sum(acc, A.abort_flag,
                        [&](const double(&t)[1]) { persist_step(A, P, st, t[0], sh.stop != 0); }))
                goto out;
        } else {
            // Richardson: x += omega r; r = b - A x
            const double omega = st.omega;
            for (int s = s_lo + warp; s < s_hi; s += kPWarps) {
                const int row = 32 * s + lane;
                if (row < n) x[row] = fma_t(omega, rl[row - base], x[row]);
            }
            if (!gs.barrier()) goto out;
            double acc[1] = {0.0};
            for (int s = s_lo + warp; s < s_hi; s += kPWarps) {
                const int row = 32 * s + lane;
                const double t = product(A.s_val, s, x);
                if (row < n) {
                    const double ri = b[row] - t;
                    rl[row - base] = ri;
                    acc[0] = fma_t(ri, ri, acc[0]);
                }
            }
            if (!gs.sum(acc, A.abort_flag,
                        [&](const double(&t)[1]) { persist_step(A, P, st, t[0], sh.stop != 0); }))
                goto out;
        }
    }
    // the last step of CG still has to reach x
    if (Tr::kCgLike && st.k > 0) {
        const double xi = st.xi;
        const double *p = A.p[0];
        for (int s = s_lo + warp; s < s_hi; s += kPWarps) {
            const int row = 32 * s + lane;
            if (row < n) x[row] = fma_t(xi, p[row], x[row]);
        }
    }
out:
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        DevState *o = P.out;
        o->nf = st.nf;
        o->norm0 = st.norm0;
        o->norm = st.norm;
        o->omega = st.omega;
        o->lambda_max = st.lambda;
        o->k = st.k;
        o->status = sh.fail ? CF_TIMEOUT : st.status;
        o->flags = sh.fail;
    }
    gs.leave();
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
template <int FMT>
static const void *persist_kernel(int solver)
{
    switch (solver) {
    case CF_CG: return (const void *)k_persist<CF_CG, FMT>;
    case CF_PCG: return (const void *)k_persist<CF_PCG, FMT>;
    case CF_JACOBI: return (const void *)k_persist<CF_JACOBI, FMT>;
    case CF_RICHARDSON: return (const void *)k_persist<CF_RICHARDSON, FMT>;
    case CF_MR: return (const void *)k_persist<CF_MR, FMT>;
    case CF_MRJACOBI:
    case CF_MRS: return (const void *)k_persist<CF_MRJACOBI, FMT>;
    case CF_JMR: return (const void *)k_persist<CF_JMR, FMT>;
    default: return nullptr;
    }
}

// The kernel of a solve over the SELL-32 copy (faster than the multi-kernel
// loop at every size, see the top of the file), or null where the loop runs:
// CSR matrices (their staging buffers), BiCG's fast order, devices without
// cooperative launches or with more SMs than the partial sums are sized for.
const void *persist_kernel_for(Context *ctx, int solver, int format)
{
    const void *k = format == kSellC ? persist_kernel<kSellC>(solver)
                    : format == kSellD ? persist_kernel<kSellD>(solver)
                    : format == kSell  ? persist_kernel<kSell>(solver)
                                       : nullptr;
    if (!k || ctx->sm_count > kPMaxGrid) return nullptr;
    if (ctx->coop_ok < 0) {
        int coop = 0;
        if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device) != cudaSuccess) {
            cudaGetLastError();
            coop = 0;
        }
        ctx->coop_ok = coop;
    }
    if (!ctx->coop_ok) return nullptr;
    return k;
}

// Shared memory a block may use for its private vectors (q and r).  At most
// this much, so that the rest of the 256 KB stays L1 for the gathers.
#ifndef CF_PERSIST_LOCAL_BYTES
#define CF_PERSIST_LOCAL_BYTES (96 * 1024)
#endif

void launch_persist(Context *ctx, const void *kernel, int solver, const SolveArgs &A, const DevState &S, int l1,
                    DevState *out)
{
    PersistArgs P;
    std::memset(&P, 0, sizeof(P));
    const size_t part = sizeof(double) * 2 * kPMaxNV * kPMaxGrid;
    if (ctx->persist.bytes == 0) {
        ctx->persist.ensure(part + 64);
        CF_CUDA(cudaMemsetAsync(ctx->persist.ptr, 0, part + 64, ctx->stream));
    }
    P.g.part = ctx->persist.as<double>();
    P.g.count = reinterpret_cast<uint32_t *>(static_cast<char *>(ctx->persist.ptr) + part);
    P.g.stop = reinterpret_cast<int32_t *>(P.g.count + 4);
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
    // at least four slices (one warp per sub-partition) per block
    const int grid = std::max(1, std::min(ctx->sm_count, (A.n_slices + 3) / 4));
    const int local_rows = 32 * ((A.n_slices + grid - 1) / grid);
    const bool two = solver == CF_CG || solver == CF_PCG || solver == CF_MRJACOBI || solver == CF_MRS;
    size_t smem = sizeof(double) * (size_t)local_rows * (two ? 2 : 1);
    P.local_rows = smem <= CF_PERSIST_LOCAL_BYTES && solver != CF_JACOBI ? local_rows : 0;
    if (P.local_rows == 0) smem = 0;
    if (smem > 48 * 1024)
        CF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    SolveArgs a = A;
    void *args[] = {&a, &P};
    CF_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kPBlock), args, smem, ctx->stream));
}

// after a solve whose blocks gave up waiting: the arrival counter is not zero
void persist_reset(Context *ctx) { ctx->persist.release(); }

} // namespace cf
