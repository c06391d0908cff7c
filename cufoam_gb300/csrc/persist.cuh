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
constexpr int kPBlock = 1024;
constexpr int kPWarps = kPBlock / 32;
constexpr int kPMaxNV = 4;
constexpr int kPMaxGrid = 192;         // blocks (SMs) the partial sums are sized for

// polls of the grid barrier before a block gives up (about half a
// microsecond each: tens of seconds); the solve then ends with CF_TIMEOUT
#ifndef CF_PERSIST_POLL_LIMIT
#define CF_PERSIST_POLL_LIMIT (1 << 25)
#endif
constexpr int kPollLimit = CF_PERSIST_POLL_LIMIT;

struct PersistGrid {
    uint32_t *count;       // arrivals since the launch (0 between launches)
    double *part;          // [2][kPMaxNV][kPMaxGrid] block partials, by parity
    int32_t *stop;         // [2] block 0's stop request (time limit), by parity
};

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
    // unit of the grid: 2^(emax - 1023 - 52 - 10)
    int ex = (int)emax - 1023 - 62;
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
    const unsigned long long out = ((unsigned long long)(ex + 63 + 1022) << 52) + r;
    return __longlong_as_double((long long)(out | (neg ? 1ull << 63 : 0ull)));
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

struct PersistShared {
    double w[kPMaxNV][kPWarps];
    double tot[kPMaxNV];
    int32_t fail;          // the barrier gave up
    int32_t stop;          // block 0 asked for an early end
};

// The grid-wide state of one block: every thread holds a copy.
struct PersistSync {
    PersistGrid g;
    PersistShared *sh;
    uint32_t epoch;        // barriers passed
    uint32_t red;          // sums done

    __device__ __forceinline__ void init(const PersistGrid &g_, PersistShared *sh_)
    {
        g = g_;
        sh = sh_;
        epoch = 0;
        red = 0;
        if (threadIdx.x == 0) {
            sh->fail = 0;
            sh->stop = 0;
        }
        __syncthreads();
    }

    // thread 0: arrive (releasing the block's writes) and wait for all blocks
    __device__ __forceinline__ void arrive_wait()
    {
        red_release(g.count);
        const uint32_t want = (epoch + 1) * gridDim.x;
        int n = 0;
        while ((int32_t)(ld_acquire(g.count) - want) < 0)
            if (++n > kPollLimit) {
                sh->fail = 1;
                break;
            }
    }

    // all of the grid's writes before it are visible after it; false: gave up
    __device__ __forceinline__ bool barrier()
    {
        __syncthreads();
        if (threadIdx.x == 0) arrive_wait();
        ++epoch;
        __syncthreads();
        return !sh->fail;
    }

    // Sums over the grid: totals in sh->tot for every thread, after
    // `post(tot)` ran in thread 0 (the step logic: the same in every block).
    // Also a grid barrier.  `abort_flag` (block 0 reads it) ends the solve.
    template <int NV, class Post>
    __device__ __forceinline__ bool sum(const double (&v)[NV], const volatile int32_t *abort_flag, Post post)
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int G = gridDim.x;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const double t[1] = {v[i]};
            const double s = warp_sum_fixed<1>(t);
            if (lane == 0) sh->w[i][warp] = s;
        }
        __syncthreads();
        if (warp == 0) {
            double *part = g.part + (size_t)(red & 1) * kPMaxNV * kPMaxGrid;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const double t[1] = {sh->w[i][lane]};
                const double s = warp_sum_fixed<1>(t);
                if (lane == 0) part[i * kPMaxGrid + blockIdx.x] = s;
            }
            if (lane == 0) {
                if (blockIdx.x == 0) g.stop[red & 1] = abort_flag ? *abort_flag : 0;
                arrive_wait();
            }
            __syncwarp();
            constexpr int kPer = kPMaxGrid / 32;
            double s[NV];
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                double t[kPer];
#pragma unroll
                for (int u = 0; u < kPer; ++u) {
                    const int b = lane + 32 * u;
                    t[u] = b < G ? ld_cg(part + i * kPMaxGrid + b) : 0.0;
                }
                s[i] = warp_sum_fixed<kPer>(t);
            }
            if (lane == 0) {
                sh->stop = ld_cg(g.stop + (red & 1));
#pragma unroll
                for (int i = 0; i < NV; ++i) sh->tot[i] = s[i];
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

} // namespace cf
