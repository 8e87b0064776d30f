// Reproducible compensated sum of per-ring partial sums (disk force, mass).
#pragma once

#include <cuda_runtime.h>

// The mean of a ring's n values by a block of 128 threads, eight loads of a
// thread in flight; complete in every thread's return value.  A value of the
// first one's sign and exponent differs from it by a whole number of units in
// its last place, the difference of the two bit patterns: those are summed as
// integers, exactly; only blocks of eight with another take FP64 additions (1.6 per
// clock and SM, also where a predicate is off: 2048 x 6144 cells in 55 us with a
// choice per value, in 22 with one per block).
__device__ __forceinline__ double block_row_mean(const double *__restrict__ v, int n)
{
    __shared__ double part[4];
    const double v0 = v[0];
    const long long b0 = __double_as_longlong(v0);
    const int top = (int)(b0 >> 52), e = top & 0x7ff;
    const bool finite = e != 0x7ff;
    long long ulps = 0;
    double other = 0.0;
    for (int j = threadIdx.x; j < n; j += 8 * 128) {
        long long u[8];
        bool same = finite;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int c = j + k * 128;
            const long long b = c < n ? __double_as_longlong(v[c]) : b0;
            same = same && (int)(b >> 52) == top;
            u[k] = b - b0;
        }
        if (same) {
#pragma unroll
            for (int k = 0; k < 8; ++k) ulps += u[k];
        } else {
#pragma unroll 1
            for (int c = j; c < n && c < j + 8 * 128; c += 128) other += v[c] - v0;
        }
    }
    const double ulp = ldexp(top < 0 ? -1.0 : 1.0, (e > 1 ? e : 1) - 1075);
    double s = other + (double)ulps * ulp;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    __syncthreads();  // part of a call before this one has been read
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    return v0 + ((part[0] + part[1]) + (part[2] + part[3])) / (double)n;
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
    if (threadIdx.x == 0) {
        for (int k = 1; k < kReduceThreads / 32; ++k)
            add_compensated(s, c, sums[0][k], sums[1][k]);
        out[w] = s - c;
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
