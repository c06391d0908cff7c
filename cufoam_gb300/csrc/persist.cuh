// persist.cuh -- building blocks of the grid-persistent solves: one
// cooperative launch of one block per SM runs a whole solve, with a grid
// barrier where the multi-kernel loop has a kernel boundary.
//
// A block owns a contiguous range of 32-row slices and a thread the same
// rows in every pass, so only the vector the product gathers crosses
// blocks.  Every block sums the block partials itself, in the same order,
// and runs the same step logic on the same bits: all take the same branch.
#pragma once

#include "solver_common.cuh"

namespace cf {

// One block of 1,024 threads per SM: 64 registers per thread, as the SpMV
// passes of the multi-kernel loop have (four blocks of 256), and a quarter
// of their arrivals at the grid barrier.  Measured on GB300 (152 SMs): 1.2
// us per barrier with 152 arrivals, 2.1 us with 608.
// (fewer warps where a block has fewer slices)
constexpr int kPBlock = 1024;
constexpr int kPWarps = kPBlock / 32;
constexpr int kPMaxNV = 4;
constexpr int kPMaxGrid = 192;         // blocks (SMs) the partial sums are sized for

struct PersistGrid {
    uint32_t *count;       // arrivals since the launch (0 between launches)
    double *part;          // [2][kPMaxNV][kPMaxGrid] block partials, by parity
    int32_t *stop;         // [2] block 0's stop request (time limit), by parity
    int32_t poll_limit;    // polls of a wait before its block gives up
};

// (hi 2^44 + mid 2^22 + lo) 2^ex, rounded once: the limbs' sums of a warp, lo and
// mid below 2^32, |hi| below 2^31.  ANY: a result that may leave the normal range
// (the check costs a grid sum 0.1 us)
template <bool ANY>
__device__ __forceinline__ double fixed_to_double(uint32_t lo, uint32_t mid, int32_t hi, int ex)
{
    // value = t 2^44 + f, 0 <= f < 2^44, then sign and magnitude
    unsigned long long f = (unsigned long long)lo + ((unsigned long long)mid << 22);
    long long t = (long long)hi + (long long)(f >> 44);
    f &= (1ull << 44) - 1;
    const bool neg = t < 0;
    if (neg) {
        t = -t;
        if (f) {
            t -= 1;
            f = (1ull << 44) - f;
        }
    }
    unsigned long long m;
    const int k = 64 - __clzll(t);           // bits of t (0 when it vanished)
    if (k > 20) {
        // more than 64 bits in all: drop the lowest k - 20, keeping a sticky bit
        const int d = k - 20;
        m = ((unsigned long long)t << (44 - d)) | (f >> d);
        if (f & ((1ull << d) - 1)) m |= 1;
        ex += d;
    } else {
        m = ((unsigned long long)t << 44) | f;
    }
    if (m == 0) return 0.0;
    const int z = __clzll(m);
    m <<= z;                                 // leading bit at 63
    ex -= z;
    // round to 53 bits, ties to even (a carry moves into the exponent)
    const unsigned long long rest = m & 0x7ffull;
    unsigned long long r = m >> 11;
    if (rest > 0x400ull || (rest == 0x400ull && (r & 1))) ++r;
    if (ANY && (ex < -1000 || ex > 900)) return scalbn((neg ? -1.0 : 1.0) * (double)r, ex + 11);
    const unsigned long long out = ((unsigned long long)(ex + 63 + 1022) << 52) + r;
    return __longlong_as_double((long long)(out | (neg ? 1ull << 63 : 0ull)));
}

// ---------------------------------------------------------------------------
// Warp sum of doubles in fixed point: every lane gets the same bits.
//
// Each value is placed on a common grid, 10 bits below the last bit of the
// largest one, as a 64-bit integer; three 22-bit limbs are summed over the
// warp by integer reductions and the total is rounded once.  On GB300 a
// warp-wide FP64 addition holds its sub-partition's FP64 unit for 64 cycles,
// so a shuffle tree in 8 warps of a sub-partition takes 5 * 8 * 64 = 2,560
// cycles; the integer form runs on the ALU.  The error is the truncation of
// 32 K terms below 2^-10 of the largest value's last bit (at most 1/32 K of
// it, K terms per lane) plus one rounding -- less than the 5 roundings of
// the tree.  Values whose largest exponent is outside [2^-900, 2^900],
// infinities and NaN take the tree.
// ---------------------------------------------------------------------------
template <int K>
__device__ __forceinline__ double warp_sum_fixed(const double (&v)[K])
{
    uint32_t e[K], emax = 0;
#pragma unroll
    for (int u = 0; u < K; ++u) {
        e[u] = ((uint32_t)__double2hiint(v[u]) >> 20) & 0x7ffu;
        emax = max(emax, e[u]);
    }
    emax = __reduce_max_sync(kFull, emax);
    if (emax < 123u || emax > 1923u) {   // (uniform) zero, tiny, huge or non-finite
        double s = v[0];
#pragma unroll
        for (int u = 1; u < K; ++u) s += v[u];
        // all zero, as where a source is zero: MR step at 219k rows 15.9 -> 12.5 us
        if (emax == 0u && !__any_sync(kFull, s != 0.0)) return 0.0;
#pragma unroll
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
        return s;
    }
    uint32_t lo = 0, mid = 0;
    int32_t hi = 0;
#pragma unroll
    for (int u = 0; u < K; ++u) {
        const long long bits = __double_as_longlong(v[u]);
        const uint32_t sh = emax - e[u];
        unsigned long long m = ((unsigned long long)bits & 0xfffffffffffffull) | (e[u] ? 1ull << 52 : 0ull);
        m = sh < 63u ? (m << 10) >> sh : 0ull;
        const long long s = bits < 0 ? -(long long)m : (long long)m;
        lo += (uint32_t)s & 0x3fffffu;
        mid += (uint32_t)(s >> 22) & 0x3fffffu;
        hi += (int32_t)(s >> 44);
    }
    lo = __reduce_add_sync(kFull, lo);     // < 32 K 2^22
    mid = __reduce_add_sync(kFull, mid);
    hi = __reduce_add_sync(kFull, hi);     // |hi| < 32 K 2^19
    return fixed_to_double<false>(lo, mid, hi, (int)emax - 1023 - 62);   // unit: 2^(emax - 1023 - 52 - 10)
}

// ---------------------------------------------------------------------------
// Dot products in fixed point.  A thread's sum of products is a 64-bit integer
// on a grid that follows its largest product, each product the upper 64 bits of
// the 106-bit product of the mantissas: exact to 2^-62, added without rounding
// except for bits below 2^(head - 63) of the largest one (head: bits kept free
// for the sum, log2 of the terms per thread).  FP64 FMA chains round every
// addition to 2^-53 of the sum.
//
// Why: on GB300 an FP64 operation holds a sub-partition's FP64 unit for 64
// cycles per warp, and the unit bounds the passes at large sizes; the integer
// form is about 30 instructions on the other pipes, beside the FP64 work.
// Measured, us per step at 0.3M / 0.9M / 2.1M rows (7-point), FMA chains -> here:
// MR 15.1 -> 14.2 / 27.2 -> 24.5 / 55.4 -> 49.0, MRJacobi 15.6 -> 14.3 / 29.5 ->
// 26.5 / 59.4 -> 53.9, Jacobi 9.7 -> 9.5 / 22.0 -> 21.1 / 46.8 -> 44.6.
// ---------------------------------------------------------------------------
struct FixedDot {
    static constexpr int kEmpty = -100000, kFloat = 100000;
    long long acc = 0;     // the sum in units of 2^(e + head - 2108); in kFloat mode a double's bits
    int e = kEmpty;        // largest ea + eb (biased exponents) so far

    __device__ __forceinline__ void add(double a, double b, int head)
    {
        const long long ab = __double_as_longlong(a), bb = __double_as_longlong(b);
        const uint32_t ea = (uint32_t)(ab >> 52) & 0x7ffu, eb = (uint32_t)(bb >> 52) & 0x7ffu;
        if (ea - 1u >= 0x7feu || eb - 1u >= 0x7feu || e == kFloat) {   // zero, subnormal, infinity or NaN
            // a term 0, inline: whole regions of a vector may be zero
            if ((2 * ab == 0 && eb < 0x7ffu) || (2 * bb == 0 && ea < 0x7ffu)) return;
            *this = slow(*this, a, b, head);
            return;
        }
        const unsigned long long h = __umul64hi(((unsigned long long)ab << 11) | (1ull << 63),
                                                ((unsigned long long)bb << 11) | (1ull << 63));
        const int s = (int)(ea + eb);
        if (s > e) {
            const int d = s - e;
            acc >>= d < 63 ? d : 63;
            e = s;
        }
        const int sh = e - s + head;
        const long long q = sh < 64 ? (long long)(h >> sh) : 0ll;
        acc += (ab ^ bb) < 0 ? -q : q;
    }
    __device__ double value(int head) const
    {
        if (e == kFloat) return __longlong_as_double(acc);
        return e == kEmpty ? 0.0 : scalbn((double)acc, e + head - 2108);
    }
    // by value: the accumulator stays in registers around the call
    static __device__ __noinline__ FixedDot slow(FixedDot f, double a, double b, int head)
    {
        const double t = fma_t(a, b, f.value(head));
        f.acc = __double_as_longlong(t);
        f.e = kFloat;
        return f;
    }
    // the warp's sum, the same bits in every lane
    __device__ __forceinline__ double warp_sum(int head) const
    {
        const int emax = __reduce_max_sync(kFull, e);
        if (emax == kFloat) {   // (uniform)
            double s = value(head);
#pragma unroll
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
            return s;
        }
        if (emax == kEmpty) return 0.0;
        const int d = emax - e;
        const long long s = acc >> (d < 63 ? d : 63);
        const uint32_t lo = __reduce_add_sync(kFull, (uint32_t)s & 0x3fffffu);
        const uint32_t mid = __reduce_add_sync(kFull, (uint32_t)(s >> 22) & 0x3fffffu);
        const int32_t hi = __reduce_add_sync(kFull, (int32_t)(s >> 44));
        return fixed_to_double<true>(lo, mid, hi, emax + head - 2108);
    }
};

// the same interface over an FP64 FMA chain
struct PlainDot {
    double v = 0.0;
    __device__ __forceinline__ void add(double a, double b, int) { v = fma_t(a, b, v); }
    __device__ __forceinline__ double warp_sum(int) const
    {
        const double t[1] = {v};
        return warp_sum_fixed<1>(t);
    }
};
__device__ __forceinline__ double warp_total(double v, int)
{
    const double t[1] = {v};
    return warp_sum_fixed<1>(t);
}
template <class D>
__device__ __forceinline__ double warp_total(const D &d, int head)
{
    return d.warp_sum(head);
}

// ---------------------------------------------------------------------------
// grid barrier and grid sums
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release(uint32_t *p)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}

// Systems up to this many rows run in one cluster of up to 16 blocks: CG step
// 5.4 us against 8.1 on the grid at 4,096 rows, 6.7 against 8.1 at 8,100, 8.6
// against 8.3 at 12,100.
#ifndef CF_PERSIST_CLUSTER_ROWS
#define CF_PERSIST_CLUSTER_ROWS 10240
#endif

constexpr int kPClusterMax = 16;       // blocks of a cluster
static_assert(CF_PERSIST_CLUSTER_ROWS % (32 * kPClusterMax) == 0, "whole warps");

// SLOTS: room for the warp sums of every block of a cluster, by parity
// (1 where the sums go through global memory)
template <int SLOTS> struct PersistShared {
    double w[kPMaxNV][kPWarps];
    double slot[2][kPMaxNV][SLOTS];
    int32_t slot_stop[2];
    int32_t fail;              // this block gave up waiting at the grid barrier
    int32_t stop;              // block 0 asked for an early end
};

// the block's sums of v in s (valid in warp 0)
template <int NV, class T>
__device__ __forceinline__ void block_sum_fixed(const T (&v)[NV], int head, PersistShared<1> *sh, double (&s)[NV])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const double x = warp_total(v[i], head);
        if (lane == 0) sh->w[i][warp] = x;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const double t[1] = {lane < nw ? sh->w[i][lane] : 0.0};
            s[i] = warp_sum_fixed<1>(t);
        }
    }
}

// ---------------------------------------------------------------------------
// The two scopes a solve runs in.  Both offer
//   barrier()  all blocks' writes before it are visible after it;
//   sum(v, abort_flag, post)  sums over all blocks (doubles, or a dot product's
//              accumulators with their `head`); thread 0 of every block
//              runs post(totals) (the step logic, the same bits everywhere)
//              before any thread goes on.  Also a barrier.  `abort_flag`,
//              read by block 0, arrives in sh->stop.
// and return false when a wait gave up (grid only).  The block then leaves at
// once, without its share of the answer, while block 0 may have seen every
// arrival: each block reports its own failure (report_fail), and any of them
// makes the solve a CF_TIMEOUT.
// ---------------------------------------------------------------------------
struct GridSync {
    static constexpr bool kCluster = false;
    static constexpr int kThreads = kPBlock;
    using Shared = PersistShared<1>;
    PersistGrid g;
    Shared *sh;
    uint32_t epoch;        // barriers passed
    uint32_t red;          // sums done

    __device__ __forceinline__ GridSync(const PersistGrid &g_, Shared *sh_) : g(g_), sh(sh_), epoch(0), red(0)
    {
        if (threadIdx.x == 0) {
            sh->fail = 0;
            sh->stop = 0;
        }
        __syncthreads();
    }
    __device__ __forceinline__ int rank() const { return blockIdx.x; }
    __device__ __forceinline__ int blocks() const { return gridDim.x; }

    // thread 0: arrive (releasing the block's writes) and wait for all blocks
    __device__ __forceinline__ void arrive_wait()
    {
        red_release(g.count);
        const uint32_t want = (epoch + 1) * gridDim.x;
        int n = 0;
        while ((int32_t)(ld_acquire(g.count) - want) < 0)
            if (++n > g.poll_limit) {
                sh->fail = 1;
                break;
            }
    }

    __device__ __forceinline__ bool barrier()
    {
        __syncthreads();
        if (threadIdx.x == 0) arrive_wait();
        ++epoch;
        __syncthreads();
        return !sh->fail;
    }

    template <int NV, class T, class Post>
    __device__ __forceinline__ bool sum(const T (&v)[NV], const volatile int32_t *abort_flag, Post post, int head = 0)
    {
        const int lane = threadIdx.x & 31;
        const int G = gridDim.x;
        double s[NV];
        block_sum_fixed(v, head, sh, s);
        if (threadIdx.x < 32) {
            double *part = g.part + (size_t)(red & 1) * kPMaxNV * kPMaxGrid;
            if (lane == 0) {
#pragma unroll
                for (int i = 0; i < NV; ++i) part[i * kPMaxGrid + blockIdx.x] = s[i];
                if (blockIdx.x == 0) g.stop[red & 1] = abort_flag ? *abort_flag : 0;
                arrive_wait();
            }
            __syncwarp();
            constexpr int kPer = kPMaxGrid / 32;
            double t[NV][kPer];
#pragma unroll
            for (int i = 0; i < NV; ++i)
#pragma unroll
                for (int u = 0; u < kPer; ++u) {
                    const int b = lane + 32 * u;
                    t[i][u] = b < G ? ld_cg(part + i * kPMaxGrid + b) : 0.0;
                }
            const int32_t stop = abort_flag ? ld_cg(g.stop + (red & 1)) : 0;
#pragma unroll
            for (int i = 0; i < NV; ++i) s[i] = warp_sum_fixed<kPer>(t[i]);
            if (lane == 0) {
                sh->stop = stop;
                post(s);
            }
        }
        ++epoch;
        ++red;
        __syncthreads();
        return !sh->fail;
    }

    // the last block to leave zeroes the counter for the next launch
    __device__ __forceinline__ void leave()
    {
        __syncthreads();
        if (threadIdx.x == 0 && !sh->fail) {
            const uint32_t old = atomicAdd(g.count, 1u);
            if (old == epoch * gridDim.x + gridDim.x - 1) *g.count = 0u;
        }
    }
};

// one thread-block cluster: the hardware barrier, sums through distributed
// shared memory
struct ClusterSync {
    static constexpr bool kCluster = true;
    // a warp per slice of the largest system a cluster takes: more registers each
    static constexpr int kThreads = CF_PERSIST_CLUSTER_ROWS / kPClusterMax;
    using Shared = PersistShared<kPClusterMax * kPWarps>;
    Shared *sh;
    uint32_t red;
    uint32_t me, n;

    __device__ __forceinline__ ClusterSync(const PersistGrid &, Shared *sh_) : sh(sh_), red(0)
    {
        asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(me));
        asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
        if (threadIdx.x == 0) {
            sh->fail = 0;
            sh->stop = 0;
        }
        __syncwarp();
        // every block runs before a peer's first store into its shared memory
        // (the first sum stores before its own barrier); 0.5 us per solve
        barrier();
    }
    __device__ __forceinline__ int rank() const { return (int)me; }
    __device__ __forceinline__ int blocks() const { return (int)n; }
    __device__ __forceinline__ bool barrier()
    {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        return true;
    }
    template <class T>
    __device__ __forceinline__ uint32_t remote(const T *p, uint32_t rank) const
    {
        uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
        return r;
    }
    template <int K> static __device__ __forceinline__ double sum_slots(const double *w, int m)
    {
        const int lane = threadIdx.x & 31;
        double t[K];
#pragma unroll
        for (int u = 0; u < K; ++u) t[u] = lane + 32 * u < m ? w[lane + 32 * u] : 0.0;
        return warp_sum_fixed<K>(t);
    }
    // Every warp stores its sum into every block's shared memory; after the
    // cluster barrier warp 0 of each block adds up what it has (no second
    // stage, no remote loads).
    template <int NV, class T, class Post>
    __device__ __forceinline__ bool sum(const T (&v)[NV], const volatile int32_t *abort_flag, Post post, int head = 0)
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
        const int par = red & 1;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const double x = warp_total(v[i], head);
            if (lane < (int)n)
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote(&sh->slot[par][i][me * nw + warp],
                                                                              (uint32_t)lane)),
                             "d"(x)
                             : "memory");
        }
        if (abort_flag && me == 0 && warp == 0 && lane < (int)n) {
            const int32_t stop = *abort_flag;
            asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(remote(&sh->slot_stop[par], (uint32_t)lane)),
                         "r"(stop)
                         : "memory");
        }
        barrier();
        if (threadIdx.x < 32) {
            const int m = (int)n * nw;
            double s[NV];
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const double *w = sh->slot[par][i];
                s[i] = m <= 128 ? sum_slots<4>(w, m) : m <= 256 ? sum_slots<8>(w, m) : sum_slots<16>(w, m);
            }
            if (lane == 0) {
                sh->stop = abort_flag ? sh->slot_stop[par] : 0;
                post(s);
            }
        }
        ++red;
        __syncthreads();
        return true;
    }
    // no block leaves while a peer may still read its shared memory
    __device__ __forceinline__ void leave() { barrier(); }
};

// out->flags (zeroed by the host before the launch): some block gave up waiting
__device__ __forceinline__ void report_fail(int32_t fail, DevState *out)
{
    if (threadIdx.x == 0 && fail) out->flags = 1;
}

// a / b with the correctly rounded reciprocal rb = 1 / b at hand: the
// rounding of a division (Markstein: one residual step from a correctly
// rounded reciprocal), three dependent FP64 operations instead of about ten
__device__ __forceinline__ double div_by_reciprocal(double a, double b, double rb)
{
    const uint32_t ea = ((uint32_t)__double2hiint(a) >> 20) & 0x7ffu, eb = ((uint32_t)__double2hiint(b) >> 20) & 0x7ffu;
    // zero, not finite, or beyond 2^+-400, where the quotient may leave the normal range
    if (ea - 623u > 800u || eb - 623u > 800u) return a / b;
    const double q = __dmul_rn(a, rb);
    return __fma_rn(__fma_rn(-q, b, a), rb, q);
}

// ---------------------------------------------------------------------------
// rows over slots in shared memory (cp, vp: this lane's first slot): the
// chain of sell_slice_at in the same order
// ---------------------------------------------------------------------------
template <class V, int M, class G>
__device__ __forceinline__ void local_batch(const int32_t *cp, const V *vp, G g, V &acc)
{
    V v[M], x[M];
#pragma unroll
    for (int u = 0; u < M; ++u) x[u] = g(cp[32 * u]);
#pragma unroll
    for (int u = 0; u < M; ++u) v[u] = vp[32 * u];
#pragma unroll
    for (int u = 0; u < M; ++u) acc = fma_t(v[u], x[u], acc);
}
template <class V, int B, class G>
__device__ __forceinline__ void local_tail(int r, const int32_t *cp, const V *vp, G g, V &acc)
{
    if constexpr (B > 1) {
        if (r == B - 1) {
            local_batch<V, B - 1>(cp, vp, g, acc);
            return;
        }
        local_tail<V, B - 1>(r, cp, vp, g, acc);
    }
}
template <class V, int B, class G>
__device__ __forceinline__ V local_slice(const int32_t *cp, const V *vp, int len, G g)
{
    V acc = V(0);
    int t0 = 0;
    for (; t0 + B <= len; t0 += B) local_batch<V, B>(cp + 32 * t0, vp + 32 * t0, g, acc);
    local_tail<V, B>(len - t0, cp + 32 * t0, vp + 32 * t0, g, acc);
    return acc;
}

// ---------------------------------------------------------------------------
// host side, shared by the FP64 and the mixed-precision solves
// ---------------------------------------------------------------------------
enum { kScopeGrid = 0, kScopeGridLocal = 1, kScopeCluster = 2 };

// Dynamic shared memory of a block: at most this much in all, and at most
// CF_PERSIST_VEC_BYTES for vectors alone when the matrix streams from L2 or
// HBM (the rest of the SM's 256 KB is the L1 of the gathers).
#ifndef CF_PERSIST_LOCAL_BYTES
#define CF_PERSIST_LOCAL_BYTES (200 * 1024)
#endif
#ifndef CF_PERSIST_VEC_BYTES
#define CF_PERSIST_VEC_BYTES (144 * 1024)
#endif
// The dynamic limit of a persistent kernel: one value for all its solves.  (A
// kernel's limit belongs to the function on the device, not to a context: a
// solve that set its own size could lower it under another thread's launch.)
constexpr size_t persist_smem_limit(bool cluster)
{
    const size_t most = CF_PERSIST_VEC_BYTES > CF_PERSIST_LOCAL_BYTES ? CF_PERSIST_VEC_BYTES : CF_PERSIST_LOCAL_BYTES;
    return cluster ? CF_PERSIST_LOCAL_BYTES - sizeof(ClusterSync::Shared) : most;
}
// whether a cluster of kPClusterMax blocks of a single-cluster kernel can be resident
bool persist_cluster_fits(Context *ctx, const void *kernel);
// The slices of `grid` blocks over a streamed matrix: the device table of their
// first slices (null: equal numbers), and the most one of them has.
const int32_t *persist_shares(Matrix *m, int grid, int &most);
// the barrier counter and partial sums of the context
PersistGrid persist_grid(Context *ctx);
// `grid` blocks, one warp per slice up to 32, cooperative or as one cluster
void launch_persist_kernel(Context *ctx, const void *kernel, bool cluster, int grid, int slices_per_block,
                           size_t smem, void **args);

} // namespace cf
