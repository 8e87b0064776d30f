// Sums over a block: ring means, the disk force's terms, and the reproducible
// compensated sum of per-ring partial sums.
#pragma once

#include "fp64_pair.cuh"

#include <cuda_runtime.h>

// The mean of a ring's n values by the block (at least 128 threads), complete in
// every thread's return value.  A value of the first one's sign and exponent
// differs from it by a whole number of units in its last place, the difference of
// the two bit patterns: those are summed as integers, exactly; only blocks of
// eight with another take FP64 additions (1.6 per clock and SM, also where a
// predicate is off: 2048 x 6144 cells in 55 us with a choice per value, in 22 with
// one per block).  n <= 2^18, or all take them (the integers' range).
__device__ __forceinline__ double block_row_mean(const double *__restrict__ v, int n)
{
    __shared__ double part[33], part_other[32];
    const int tid = threadIdx.x, bs = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const double v0 = v[0];
    const long long b0 = __double_as_longlong(v0);
    const int top = (int)(b0 >> 52), e = top & 0x7ff;
    const bool exact = e != 0x7ff && n <= 1 << 18;
    long long ulps = 0;
    int others = 0;
    double other = 0.0;
    for (int j = tid; j < n; j += 8 * bs) {
        long long u[8];
        bool same = exact;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int c = j + k * bs;
            const long long b = c < n ? __double_as_longlong(v[c]) : b0;
            same = same && (int)(b >> 52) == top;
            u[k] = b - b0;
        }
        if (same) {
#pragma unroll
            for (int k = 0; k < 8; ++k) ulps += u[k];
        } else {
#pragma unroll 1
            for (int c = j; c < n && c < j + 8 * bs; c += bs) {
                other += v[c];
                ++others;
            }
        }
    }
    double s = (double)ulps;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    const bool any = __syncthreads_or(others);  // (part of a call before this has been read)
    if (any) {
        other = fma(-(double)others, v0, other);
        for (int o = 16; o > 0; o >>= 1) other += __shfl_down_sync(0xffffffffu, other, o);
        if (lane == 0) part_other[warp] = other;
    }
    if (lane == 0) part[warp] = s;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0, to = 0.0;
        for (int w = 0; w < bs >> 5; ++w) {
            t += part[w];
            if (any) to += part_other[w];
        }
        const double ulp = ldexp(top < 0 ? -1.0 : 1.0, (e > 1 ? e : 1) - 1075);
        part[32] = v0 + (t * ulp + to) / (double)n;
    }
    __syncthreads();
    return part[32];
}

namespace fgpu {
__device__ __forceinline__ f2 pair_plus(f2 a, f2 b)
{
    const f2 s = two_sum(a.h, b.h);
    return f2{s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l))};
}
__device__ __forceinline__ f2 pair_from(f2 a, int o)
{
    return f2{__shfl_xor_sync(0xffffffffu, a.h, o), __shfl_xor_sync(0xffffffffu, a.l, o)};
}
// the sum of a lane's two cells
__device__ __forceinline__ f2 pair_halves(f2x2 s) { return pair_plus(first(s), second(s)); }
}  // namespace fgpu

// One sum over the block, a packed float pair of every thread; the value is thread
// 0's (part: a double per warp).  Three floats carry it across a warp's lanes (the
// additions of high and low parts by TwoSum, their errors in the third), FP64 across
// the warps: in two floats a large value's low part loses the other lanes' small ones
// (the mass of 60 disks within 2.1e-16 rms, not 1.4e-16); in FP64 from the threads on,
// eight additions each, the call on 512 x 1536 cells takes 2 us more.
__device__ __forceinline__ double block_pair_sum(fgpu::f2x2 v, double *part)
{
    using fgpu::f2;
    float h = v.h.x, l = v.l.x, m = 0.f;
    auto add = [&](float h2, float l2, float m2) {
        const f2 s = fgpu::two_sum(h, h2), t = fgpu::two_sum(l, l2), u = fgpu::two_sum(s.l, t.h);
        h = s.h;
        l = u.h;
        m = __fadd_rn(__fadd_rn(m, m2), __fadd_rn(t.l, u.l));
    };
    add(v.h.y, v.l.y, 0.f);
    for (int o = 16; o > 0; o >>= 1)
        add(__shfl_xor_sync(0xffffffffu, h, o), __shfl_xor_sync(0xffffffffu, l, o),
            __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = (double)h + ((double)l + (double)m);
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < blockDim.x >> 5; ++w) t += part[w];
    return t;
}

// Eight sums of every thread of the block, float pairs (hi, lo) each: the halves
// of a warp exchange four of the eight, then two, then one, so a warp adds nine
// pairs where eight separate sums would add forty (in FP64, 20 cycles an SM each,
// these took longer than a 128-cell ring's terms); the warps' sums in FP64.
// Complete in total[0 .. 7] after the call; every sum is formed along the same
// tree.
__device__ __forceinline__ void block_eight_sums(const fgpu::f2 (&v)[8], double *part, double *total)
{
    using fgpu::f2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    f2 a[4], b[2];
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = fgpu::pair_plus(b4 ? v[k + 4] : v[k],
                               fgpu::pair_from(b4 ? v[k] : v[k + 4], 16));
#pragma unroll
    for (int k = 0; k < 2; ++k) b[k] = fgpu::pair_plus(b3 ? a[k + 2] : a[k],
                               fgpu::pair_from(b3 ? a[k] : a[k + 2], 8));
    f2 s = fgpu::pair_plus(b2 ? b[1] : b[0], fgpu::pair_from(b2 ? b[0] : b[1], 4));
    s = fgpu::pair_plus(s, fgpu::pair_from(s, 2));
    s = fgpu::pair_plus(s, fgpu::pair_from(s, 1));
    // lane 4 q holds sum q (bits 4, 3, 2 of the lane: 4, 2, 1)
    if ((lane & 3) == 0) part[8 * warp + (lane >> 2)] = (double)s.h + (double)s.l;
    __syncthreads();
    if (threadIdx.x < 8) {
        double t = 0.0;
        for (int w = 0; w < blockDim.x >> 5; ++w) t += part[8 * w + threadIdx.x];
        total[threadIdx.x] = t;
    }
    __syncthreads();
}

// hi + lo with lo the compensation still to be subtracted: s + s2 exactly
// (Knuth's TwoSum) into s, the compensations added
__device__ __forceinline__ void add_compensated(double &s, double &c, double s2, double c2)
{
    const double t = s + s2;
    const double bp = t - s;
    const double e = (s - (t - bp)) + (s2 - bp);  // s + s2 = t + e exactly
    c = (c + c2) - e;
    s = t;
}

// Component w of `rows` rows of `width` partial sums, summed by a block of
// kReduceThreads threads: thread t adds rows t, t + kReduceThreads, ... with
// Kahan compensation, the threads' sums are combined along a fixed tree with
// TwoSum.  The order is fixed, so the result is the same on every run.  (One
// warp per component spends 11 us on 2046 rows, 64 dependent additions per
// lane; this 4.)
constexpr int kReduceThreads = 256;
__device__ __forceinline__ void block_compensated_rows(const double *__restrict__ partial,
                                                       int rows, int width, int w,
                                                       double *__restrict__ out)
{
    __shared__ double sums[2][kReduceThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double s = 0.0, c = 0.0;
#pragma unroll 4
    for (int r = threadIdx.x; r < rows; r += kReduceThreads) {
        const double y = partial[(size_t)r * width + w] - c;
        const double t = s + y;
        c = (t - s) - y;
        s = t;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double s2 = __shfl_down_sync(0xffffffffu, s, o);
        const double c2 = __shfl_down_sync(0xffffffffu, c, o);
        add_compensated(s, c, s2, c2);
    }
    if (lane == 0) {
        sums[0][warp] = s;
        sums[1][warp] = c;
    }
    __syncthreads();
    if (warp == 0) {
        constexpr int warps = kReduceThreads / 32;
        s = lane < warps ? sums[0][lane] : 0.0;
        c = lane < warps ? sums[1][lane] : 0.0;
        for (int o = warps / 2; o > 0; o >>= 1) {
            const double s2 = __shfl_down_sync(0xffffffffu, s, o);
            const double c2 = __shfl_down_sync(0xffffffffu, c, o);
            add_compensated(s, c, s2, c2);
        }
        if (lane == 0) out[w] = s - c;
    }
}

// Component w of `rows` rows of `width` partial sums, summed by one warp:
// lane l adds rows l, l + 32, ... with Kahan compensation, then the 32
// (sum, compensation) pairs are combined along a fixed shuffle tree with
// Knuth's TwoSum, which recovers the rounding error of each addition
// exactly.  The order of operations is fixed, so the result is the same on
// every run.  Every lane of the warp must call it with the same w.
__device__ __forceinline__ void warp_compensated_rows(const double *__restrict__ partial, int rows,
                                                      int width, int w, double *__restrict__ out)
{
    const int lane = threadIdx.x & 31;
    double s = 0.0, c = 0.0;  // the sum is s - c
    for (int r = lane; r < rows; r += 32) {
        const double y = partial[(size_t)r * width + w] - c;
        const double t = s + y;
        c = (t - s) - y;
        s = t;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double s2 = __shfl_down_sync(0xffffffffu, s, o);
        const double c2 = __shfl_down_sync(0xffffffffu, c, o);
        add_compensated(s, c, s2, c2);
    }
    if (lane == 0) out[w] = s - c;
}
