// ksum.cuh -- compensated FP64 accumulation (TwoSum / Neumaier) and the
// deterministic block reduction used by every reduction kernel.
#pragma once
#include <cuda_runtime.h>

namespace opx {

struct KSum {
    double s, c;
};
__host__ __device__ __forceinline__ void two_sum_add(KSum &a, double x) {
    double t = a.s + x;
    double z = t - a.s;
    a.c += (a.s - (t - z)) + (x - z);
    a.s = t;
}
__host__ __device__ __forceinline__ void ksum_merge(KSum &a, const KSum &b) {
    two_sum_add(a, b.s);
    a.c += b.c;
}

// NQ per-thread compensated running sums held in shared memory ([NQ][NT]
// pairs, NT = blockDim.x): they live across a whole lattice loop, where the
// registers are wanted for the site arithmetic.  A thread touches only its own
// slots, so no synchronisation is needed until the block reduction.
template <int NQ, int NT>
struct SharedKSums {
    double2 *a;
    __device__ __forceinline__ void zero() const {
#pragma unroll
        for (int q = 0; q < NQ; q++) a[q * NT + threadIdx.x] = make_double2(0.0, 0.0);
    }
    __device__ __forceinline__ void add1(int q, double x) const {
        const double2 v = a[q * NT + threadIdx.x];
        KSum k{v.x, v.y};
        two_sum_add(k, x);
        a[q * NT + threadIdx.x] = make_double2(k.s, k.c);
    }
    __device__ __forceinline__ void add(const double *p) const {
#pragma unroll
        for (int q = 0; q < NQ; q++) add1(q, p[q]);
    }
    __device__ __forceinline__ void load(KSum *acc) const {
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const double2 v = a[q * NT + threadIdx.x];
            acc[q] = KSum{v.x, v.y};
        }
    }
};

// Plain FP64 per-thread sums in shared memory ([NQ][NT]), for values that
// carry FP32 rounding already (the FP32 run sums of the paired SU(3) kernels):
// one FP64 add per column per flush.
template <int NQ, int NT>
struct SharedSums {
    double *a;
    __device__ __forceinline__ void zero() const {
#pragma unroll
        for (int q = 0; q < NQ; q++) a[q * NT + threadIdx.x] = 0.0;
    }
    __device__ __forceinline__ void add1(int q, double x) const { a[q * NT + threadIdx.x] += x; }
    __device__ __forceinline__ void load(KSum *acc) const {
#pragma unroll
        for (int q = 0; q < NQ; q++) acc[q] = KSum{a[q * NT + threadIdx.x], 0.0};
    }
};

// Sums of FP64 values over a warp or over an array on the integer pipe: a warp's
// FP64 instruction takes 65 clocks of its scheduler's FP64 lanes here, so a tree of
// them is what the end of a small reduction waits for.  The mantissas are aligned
// to the largest exponent and added as integers; the one rounding of the result
// to double follows an alignment error below it, whatever the order.

__device__ __forceinline__ unsigned long long warp_add_u64(unsigned long long x) {
    // limbs of 22, 22 and 20 bits: 32 of each fit 32 bits
    const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)x & 0x3fffffu);
    const unsigned mid = __reduce_add_sync(0xffffffffu, (unsigned)(x >> 22) & 0x3fffffu);
    const unsigned hi = __reduce_add_sync(0xffffffffu, (unsigned)(x >> 44));
    return (unsigned long long)lo + ((unsigned long long)mid << 22) + ((unsigned long long)hi << 44);
}
// the sum over the warp of v >= 0 (or not finite), on every lane
__device__ __forceinline__ double warp_sum(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int e = (int)(b >> 52);  // a sign bit makes it negative or large: not this way
    const int top = (int)__reduce_max_sync(0xffffffffu, (unsigned)e);
    if (top >= 0x7ff || top < 64) {  // not finite, negative, or too near the end of the range
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    }
    const unsigned long long m = ((b & 0xfffffffffffffULL) | 0x10000000000000ULL) << 6;  // 59 bits; e = 0 shifts out
    const int k = top - e;
    const unsigned long long t = warp_add_u64(k < 64 ? ((m >> k) + 1) >> 1 : 0ULL);  // units 2^(top - 1080)
    return (double)t * __longlong_as_double((long long)(top - 57) << 52);
}
// the sum of x[0], x[stride], ... x[(n - 1) stride] (pairs value + correction) over
// the warp, every value >= 0 (or not finite), on every lane.  512 pairs at a time,
// all of a lane's loads in flight together (one at a time, a reduction's last block
// took 20 us for 456 pairs)
__device__ __forceinline__ double warp_sum_pairs(const double *x, int n, long stride) {
    constexpr int PER = 16;
    const int lane = threadIdx.x & 31;
    KSum total{0.0, 0.0};
    for (int base = 0; base < n; base += 32 * PER) {
        double v[PER];
        unsigned top = 0;
#pragma unroll
        for (int k = 0; k < PER; k++) {
            const int b = base + 32 * k + lane;
            const double *p = x + (b < n ? b : n - 1) * stride;
            const double s = __ldcg(p), c = __ldcg(p + 1);
            v[k] = b < n ? s + c : 0.0;
        }
#pragma unroll
        for (int k = 0; k < PER; k++) {
            const unsigned e = (unsigned)((unsigned long long)__double_as_longlong(v[k]) >> 52);
            top = e > top ? e : top;
        }
        top = __reduce_max_sync(0xffffffffu, top);
        if (top >= 0x7ffu || top < 128u) {  // not finite, negative, or too near the end of the range
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < PER; k++) s += v[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            two_sum_add(total, s);
            continue;
        }
        // integer part in units of 2^(top - 1075) (512 mantissas of 53 bits fit), 32 bits below it
        unsigned long long a = 0, f = 0;
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const unsigned long long u = (unsigned long long)__double_as_longlong(v[j]);
            const unsigned k = top - (unsigned)(u >> 52);
            const unsigned long long m = (u & 0xfffffffffffffULL) | 0x10000000000000ULL;
            if (k < 64) {
                a += m >> k;
                f += k < 32 ? (m << (32 - k)) & 0xffffffffULL : (m >> (k - 32)) & 0xffffffffULL;
            }
        }
        f = warp_add_u64(f);
        a = warp_add_u64(a) + (f >> 32);
        f &= 0xffffffffULL;
        const double unit = __longlong_as_double((long long)((int)top - 52) << 52);  // 2^(top - 1075)
        two_sum_add(total, ((double)a + (double)f * 0x1p-32) * unit);
    }
    return total.s + total.c;
}

// Reduce NQ per-thread sums over a block (blockDim.x a multiple of 32, at most
// 1024).  Thread q < NQ of the block receives the block total of quantity q.
// Each thread's compensated sum collapses to one double, the lanes of a warp
// are added in a fixed shuffle tree (five roundings deep) and the warps in
// order with compensation.  The tree keeps the FP64 instruction count low: the
// FP64 pipe of this part is narrow, and a compensated shuffle tree over eleven
// columns took a fifth of a whole-lattice reduction.
template <int NQ>
__device__ __forceinline__ KSum block_reduce(KSum *acc, int &qout) {
    __shared__ double sh[NQ][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < NQ; q++) {
        double v = acc[q].s + acc[q].c;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) sh[q][warp] = v;
    }
    __syncthreads();
    KSum v{0.0, 0.0};
    qout = -1;
    if (threadIdx.x < NQ) {
        const int q = threadIdx.x;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) two_sum_add(v, sh[q][w]);
        qout = q;
    }
    return v;
}

}  // namespace opx
