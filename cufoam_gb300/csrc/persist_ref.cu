// persist_ref.cu -- BiCG in the reference's summation order (its default) as
// one cooperative launch, the bits of the multi-kernel loop (solve_fp64.cu).
//
// The reference's reductions (gis/SparseSystem/kernels.h:153-199) sum the rows
// of thread s of 1,216 x 256 in row order, each block of 256 by its tree, and
// the 1,216 block sums one after the other.  Here a block of 512 threads
// stands for two of the reference's blocks at a time, the tree runs per 256
// threads, and every block forms the sequential sums itself (seq_prepare,
// seq_finish) from the 1,216 partials -- so a step needs two grid barriers
// for its sums and one before the gathers, instead of two kernels whose last
// blocks work alone.
//
// Measured on GB300 (7-point convection-diffusion, us per step, multi-kernel
// loop -> here): 22k rows 42 -> 29, 113k 57 -> 43, 893k 159 -> 148, 2.1M 271 ->
// 250; set-up of a solve 148 -> 61 us at 22k and 617 -> 456 at 2.1M.  What is
// left: the FP64 unit (a row costs 14 operations per product in the 8-lane
// order, A and A^T, and 8 more: 250,000 cycles of the 500,000 at 2.1M rows) and
// about 7 us for each of the step's two reductions.
#include "persist.cuh"

#include <algorithm>
#include <climits>
#include <cstring>

namespace cf {

struct RefArgs {
    PersistGrid g;
    double *part;            // [2][kRefNV][ref_grid]
    DevState *out;           // host-mapped: the final state
    double tolerance, rel_tol, int_bound;
    int32_t max_steps, min_steps, hist_cap, abs_tol, l1;
    int32_t ref_grid;        // the reference's blocks
};

constexpr int kRefNV = 3;
constexpr int kRefBlock = 512;                 // threads per block (128 registers each: no spills)
constexpr int kRefGroups = kRefBlock / kBlock; // the reference's blocks a block stands for at a time

struct RefState {
    double rho0, xi, theta, tol, nf, norm, norm0, xbar;
    int32_t k, done, status, x_pending;
};

struct RefShared {
    double tree[kRefNV][kRefBlock];
    double buf[kRefGroups][kSeqMax];
    double rec[kRefGroups][2 * kSeqEvents];
    SeqScratch sc[kRefGroups];
    double tot[kRefNV];
    PersistShared<1> sync;
};

// ((t0+t4)+(t2+t6)) + ((t1+t5)+(t3+t7)) of a row's 8 lanes (sell_ref_row's
// bits), all columns and values of a round of 8 slots loaded before its gathers
template <class G>
__device__ __forceinline__ double ref_row(const int32_t *cp, const double *vp, int len, int rl, G g)
{
    double t[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) t[l] = 0.0;
    for (int t0 = 0; t0 < len; t0 += 8) {
        int c[8];
        double v[8];
#pragma unroll
        for (int l = 0; l < 8; ++l)
            if (t0 + l < rl) {
                c[l] = __ldg(cp + 32 * (t0 + l));
                v[l] = __ldg(vp + 32 * (t0 + l));
            }
#pragma unroll
        for (int l = 0; l < 8; ++l)
            if (t0 + l < rl) t[l] = fma_t(v[l], g(c[l]), t[l]);
    }
    return tree8(t);
}

__global__ void __launch_bounds__(kRefBlock, 1)
    k_persist_bicg(const __grid_constant__ SolveArgs A, const __grid_constant__ RefArgs P)
{
    extern __shared__ __align__(16) unsigned char smem_[];
    RefShared &sh = *reinterpret_cast<RefShared *>(smem_);
    __shared__ RefState st;
    if (threadIdx.x == 0) {
        st = RefState{};
        st.k = -1;   // (no residual yet)
    }
    GridSync gs(P.g, &sh.sync);
    const int n = A.n, G = P.ref_grid;
    const int tid = threadIdx.x & (kBlock - 1), group = threadIdx.x / kBlock;
    const int lane = threadIdx.x & 31;
    const bool first = blockIdx.x == 0;
    uint32_t red = 0;
    double *const x = A.x, *const r = A.r[0], *const rs = A.rs, *const p = A.p[0], *const ps = A.ps[0];
    double *const q = A.q, *const qs = A.qs;
    const double *const b = A.b;
    const int stride = G * kBlock;           // rows between two of a thread's rows

    // f(row) for this thread's rows in the reference's order: block B stands for
    // the reference's blocks B, B + gridDim, ..., kRefGroups of them (a round) at
    // a time, one per group of 256 threads -- small systems fill the first of
    // the reference's blocks only, and dealt out like this they still spread
    // evenly; `end` closes a round (the tree of each group's accumulators)
    auto rows = [&](auto f, auto end) {
        for (int v0 = blockIdx.x; v0 < G; v0 += kRefGroups * gridDim.x) {
            const int vb = v0 + group * gridDim.x;
            // all lanes of a warp together (the chunk base is warp-uniform)
            if (vb < G)
                for (int64_t base = (int64_t)vb * kBlock + (tid & ~31); base < n; base += stride) f((int)base + lane);
            end(v0);
        }
    };
    // closes the round of block v0: acc of each group through the reference's
    // block tree to the partials of this reduction; acc back to zero
    auto close = [&](auto &acc, int v0) {
        const int vb = v0 + group * gridDim.x;
        constexpr int NV = sizeof(acc) / sizeof(double);
        double *part = P.part + (size_t)(red & 1) * kRefNV * G;
        if ((int64_t)v0 * kBlock >= n) {   // (uniform) a round without rows
            if (tid < NV && vb < G) part[(size_t)tid * G + vb] = 0.0;
            return;
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) sh.tree[i][threadIdx.x] = acc[i];
        __syncthreads();
        double *sm0 = &sh.tree[0][group * kBlock];
        if (tid < 128)
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                double *sm = sm0 + i * kRefBlock;
                sm[tid] = sm[tid] + sm[tid + 128];
            }
        __syncthreads();
        if (tid < 64)
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                double *sm = sm0 + i * kRefBlock;
                sm[tid] = sm[tid] + sm[tid + 64];
            }
        __syncthreads();
        if (tid < 32) {
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                double *sm = sm0 + i * kRefBlock;
                double v = sm[tid] + sm[tid + 32];
                v = v + __shfl_down_sync(kFull, v, 16);
                v = v + __shfl_down_sync(kFull, v, 8);
                v = v + __shfl_down_sync(kFull, v, 4);
                v = v + __shfl_down_sync(kFull, v, 2);
                v = v + __shfl_down_sync(kFull, v, 1);
                if (tid == 0 && vb < G) part[(size_t)i * G + vb] = v;
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NV; ++i) acc[i] = 0.0;
    };
    // all rounds closed: the sequential sums of NV values into sh.tot, then
    // post in thread 0 of every block
    auto sums = [&](int nv, const volatile int32_t *abort_flag, auto post) {
        if (first && threadIdx.x == 0) P.g.stop[red & 1] = abort_flag ? *abort_flag : 0;
        if (!gs.barrier()) return false;
        const double *part = P.part + (size_t)(red & 1) * kRefNV * G;
        for (int i0 = 0; i0 < nv; i0 += kRefGroups) {
            const int i = i0 + group;
            const bool mine = i < nv;   // (a group without a value sees an empty sum)
            seq_prepare(part + (size_t)(mine ? i : 0) * G, mine ? G : 0, sh.buf[group], sh.rec[group], &sh.sc[group],
                        tid);
            if (mine && tid < 32) {
                const double s = seq_finish(part + (size_t)i * G, G, sh.rec[group], &sh.sc[group]);
                if (lane == 0) sh.tot[i] = s;
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            sh.sync.stop = abort_flag ? ld_cg(P.g.stop + (red & 1)) : 0;
            post();
        }
        ++red;
        __syncthreads();
        return true;
    };
    auto record = [&](int k, double norm) {
        if (first && k < P.hist_cap) {
            if (A.hist) A.hist[k] = norm;
            if (A.hist_t) A.hist_t[k] = global_ns();
        }
    };
    struct Slice {
        const int32_t *cp;
        const double *v1, *v2;
        int len, rl;
    };
    auto slice = [&](int row) {
        const int s = row >> 5;
        const int o = __ldg(A.s_off + s);
        Slice c;
        c.len = (__ldg(A.s_off + s + 1) - o) >> 5;
        c.rl = row < n ? __ldg(A.ro + row + 1) - __ldg(A.ro + row) : 0;
        c.cp = A.s_col + o + lane;
        c.v1 = A.s_val + o + lane;
        c.v2 = A.s_valT + o + lane;
        return c;
    };

    // ---- normFactor and the initial residual (k_nf_sum, k_nf_dist, k_res_init)
    {
        double acc[1] = {0.0};
        rows([&](int row) { if (row < n) acc[0] = acc[0] + x[row]; }, [&](int v0) { close(acc, v0); });
        if (!sums(1, nullptr, [&] { st.xbar = sh.tot[0] / n; })) goto out;
    }
    {
        const double xbar = st.xbar;
        double acc[3] = {0.0, 0.0, 0.0};
        rows(
            [&](int row) {
                const Slice c = slice(row);
                const double Y = ref_row(c.cp, c.v1, c.len, c.rl, [&](int j) { return x[j]; });
                double Yb;
                if (!P.l1) Yb = ref_row(c.cp, c.v1, c.len, c.rl, [&](int) { return xbar; });
                else Yb = __dmul_rn(ref_row(c.cp, c.v1, c.len, c.rl, [&](int) { return 1.0; }), xbar);
                if (row < n) {
                    const double bi = b[row];
                    const double d1 = Y - Yb, d2 = bi - Yb, ri = bi - Y;
                    if (!P.l1) {
                        acc[0] = fma_t(d1, d1, acc[0]);
                        acc[1] = fma_t(d2, d2, acc[1]);
                    } else {
                        acc[0] = acc[0] + (fabs(d1) + fabs(d2));
                    }
                    r[row] = ri;
                    rs[row] = ri;
                    acc[2] = fma_t(ri, ri, acc[2]);
                }
            },
            [&](int v0) { close(acc, v0); });
        if (!sums(3, nullptr, [&] {
                const double nf = P.l1 ? sh.tot[0] + 1e-20 : sqrt(sh.tot[0]) + sqrt(sh.tot[1]) + 1e-20;
                const double norm0 = sqrt(sh.tot[2]);
                st.nf = nf;
                st.tol = P.abs_tol ? P.tolerance : P.tolerance * nf;
                if (P.rel_tol > 0.0) st.tol = fmax(st.tol, P.rel_tol * norm0);
                st.rho0 = sh.tot[2];
                st.norm0 = st.norm = norm0;
                st.xi = st.theta = 0.0;
                st.k = 0;
                st.x_pending = 0;
                record(0, norm0);
                const bool finite = isfinite(norm0);
                st.done = finite && P.max_steps >= 1 ? 0 : 1;
                st.status = !finite ? CF_NONFINITE : (norm0 > st.tol ? CF_NOT_CONVERGED : CF_OK);
            }))
            goto out;
    }

    // ---- the iterations (SolverSingleGPU.h:568-675) ---------------------------
    while (!st.done) {
        // x += xi p (the previous step), p = r + theta p, p* = r* + theta p*
        {
            const bool start = st.k == 0, pending = st.x_pending != 0;
            const double theta = st.theta, xi = st.xi;
            rows(
                [&](int row) {
                    if (row < n) {
                        double pi = r[row], psi = rs[row];
                        if (!start) {
                            const double p0 = p[row];
                            if (pending) x[row] = fma_t(xi, p0, x[row]);
                            pi = fma_t(theta, p0, pi);
                            psi = fma_t(theta, ps[row], psi);
                        }
                        p[row] = pi;
                        ps[row] = psi;
                    }
                },
                [](int) {});
            if (!gs.barrier()) goto out;
        }
        // q = A p, q* = A^T p*, (p*, q), the breakdown test
        {
            double acc[1] = {0.0};
            rows(
                [&](int row) {
                    const Slice c = slice(row);
                    const double y1 = ref_row(c.cp, c.v1, c.len, c.rl, [&](int j) { return p[j]; });
                    const double y2 = ref_row(c.cp, c.v2, c.len, c.rl, [&](int j) { return ps[j]; });
                    if (row < n) {
                        q[row] = y1;
                        qs[row] = y2;
                        acc[0] = fma_t(ps[row], y1, acc[0]);
                    }
                },
                [&](int v0) { close(acc, v0); });
            if (!sums(1, nullptr, [&] {
                    const double xi = st.rho0 / sh.tot[0];
                    st.x_pending = 0;
                    if (xi > -P.int_bound && xi < P.int_bound) {
                        st.done = 1;
                        st.status = CF_BREAKDOWN;
                    } else {
                        st.xi = xi;
                    }
                }))
                goto out;
            if (st.done) break;
        }
        // r -= xi q, r* -= xi q*, ||r||, (r, r*)
        {
            const double xi = st.xi;
            double acc[2] = {0.0, 0.0};
            rows(
                [&](int row) {
                    if (row < n) {
                        const double ri = fma_t(-xi, q[row], r[row]);
                        const double rsi = fma_t(-xi, qs[row], rs[row]);
                        r[row] = ri;
                        rs[row] = rsi;
                        acc[0] = fma_t(ri, ri, acc[0]);
                        acc[1] = fma_t(ri, rsi, acc[1]);
                    }
                },
                [&](int v0) { close(acc, v0); });
            if (!sums(2, A.abort_flag, [&] {
                    const double norm = sqrt(sh.tot[0]);
                    const int k = st.k + 1;
                    st.k = k;
                    st.norm = norm;
                    st.x_pending = 1;
                    record(k, norm);
                    bool cont = true;
                    int status = CF_NOT_CONVERGED;
                    if (norm < st.tol && k >= P.min_steps) {
                        cont = false;
                        status = CF_OK;
                    } else if (k >= P.max_steps) {
                        cont = false;
                    } else if (!isfinite(norm)) {
                        cont = false;
                        status = CF_NONFINITE;
                    }
                    if (sh.sync.stop) {
                        cont = false;
                        status = CF_TIMEOUT;
                    }
                    if (cont) {
                        const double rho1 = st.rho0;
                        st.rho0 = sh.tot[1];
                        st.theta = st.rho0 / rho1;
                    } else {
                        st.done = 1;
                        st.status = status;
                    }
                }))
                goto out;
        }
    }
    // the last step still has to reach x
    if (st.x_pending) {
        const double xi = st.xi;
        rows([&](int row) { if (row < n) x[row] = fma_t(xi, p[row], x[row]); }, [](int) {});
    }
out:
    if (first && threadIdx.x == 0) {
        DevState *o = P.out;
        o->nf = st.nf;
        o->norm0 = st.norm0;
        o->norm = st.norm;
        o->omega = 0.0;
        o->k = st.k;
        o->status = st.status;
    }
    report_fail(sh.sync.fail, P.out);
    gs.leave();
}

// Whether BiCG in the reference order runs here: over the SELL-32 copy, with
// the reference's grid within what the sequential sums take.
bool persist_ref_usable(Context *ctx, int solver, bool sell)
{
    return solver == CF_BICG && sell && ctx->ref_grid <= kSeqMax && persist_possible(ctx);
}

void launch_persist_ref(Context *ctx, const SolveArgs &A, const DevState &S, int l1, DevState *out)
{
    RefArgs P;
    std::memset(&P, 0, sizeof(P));
    P.g = persist_grid(ctx);
    ctx->persist_ref.ensure(sizeof(double) * 2 * kRefNV * (size_t)ctx->ref_grid);
    P.part = ctx->persist_ref.as<double>();
    P.out = out;
    P.tolerance = S.tolerance;
    P.rel_tol = S.rel_tol;
    P.int_bound = S.int_bound;
    P.max_steps = S.max_steps;
    P.min_steps = S.min_steps;
    P.hist_cap = S.hist_cap;
    P.abs_tol = (S.flags & kFlagAbsTol) ? 1 : 0;
    P.l1 = l1;
    P.ref_grid = ctx->ref_grid;
    SolveArgs a = A;
    void *args[] = {&a, &P};
    out->flags = 0;   // (S may be *out: read above)
    launch_persist_kernel(ctx, (const void *)k_persist_bicg, false, ctx->sm_count, kRefBlock / 32, sizeof(RefShared), args);
}

} // namespace cf
