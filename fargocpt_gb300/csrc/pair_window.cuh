// Windows of the float-pair cell kernels: a warp marches through the rings of
// one window of 64 consecutive azimuthal cells, two adjacent cells per lane as
// one packed pair (fp64_pair.cuh), and writes the 60 inner ones.  The left
// neighbour of a lane's first cell and the right neighbour of its second come
// by shuffles, the ring below from registers: a value is loaded and split into
// a pair once, where one thread per cell split it once per stencil point that
// used it, and every pair operation serves two cells.
#pragma once

#include "fp64_pair.cuh"
#include "hydro.cuh"

namespace fgpu {
namespace win {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kInner = 60;      // cells a warp writes per ring
constexpr int kThreads = 128;   // threads per block

inline int windows(int nz) { return (nz + kInner - 1) / kInner; }
// rings per march of a grid of nwin windows (kernels_kick.cu)
int march_rings(int nr, int nwin);

__device__ __forceinline__ f2x2 operator+(f2x2 a, f2x2 b) { return f2_sadd(a, b); }
__device__ __forceinline__ f2x2 operator-(f2x2 a, f2x2 b) { return f2_ssub(a, b); }
__device__ __forceinline__ f2x2 operator-(f2x2 a) { return f2_neg(a); }
__device__ __forceinline__ f2x2 operator*(f2x2 a, f2x2 b) { return f2_smul(a, b); }
__device__ __forceinline__ f2x2 operator/(f2x2 a, f2x2 b) { return f2_sdiv(a, b); }

// x s for a power of two s (exact)
__device__ __forceinline__ f2x2 sc(f2x2 x, float s)
{
    const float2 v = make_float2(s, s);
    return f2x2{vmul(x.h, v), vmul(x.l, v)};
}
// a constant the host split, on both cells
__device__ __forceinline__ f2x2 K(float2 v) { return pack(f2{v.x, v.y}); }
// a literal
__device__ __forceinline__ f2x2 P(double x) { return pack(f2_split(x)); }
// ring i's value of one of the per-ring tables
__device__ __forceinline__ f2x2 T(const Tables &t, const double *tab, int i)
{
    return K(t.ptab[(tab - t.tbase) + i]);
}

__device__ __forceinline__ f2 from_left(f2 a)
{
    return f2{__shfl_up_sync(kAll, a.h, 1), __shfl_up_sync(kAll, a.l, 1)};
}
__device__ __forceinline__ f2 from_right(f2 a)
{
    return f2{__shfl_down_sync(kAll, a.h, 1), __shfl_down_sync(kAll, a.l, 1)};
}
// the values of the left (right) neighbours of a lane's two cells
__device__ __forceinline__ f2x2 left(f2x2 a) { return pack(from_left(second(a)), first(a)); }
__device__ __forceinline__ f2x2 right(f2x2 a) { return pack(second(a), from_right(first(a))); }

// two adjacent doubles
struct d2 {
    double a, b;
};
__device__ __forceinline__ f2x2 split(d2 x) { return pack(f2_split(x.a), f2_split(x.b)); }
__device__ __forceinline__ d2 join(f2x2 x)
{
    return d2{f2_to_double(first(x)), f2_to_double(second(x))};
}
// x + dx: the FP64 values plus the joined pair increments
__device__ __forceinline__ d2 upd(d2 x, f2x2 dx)
{
    const d2 d = join(dx);
    return d2{x.a + d.a, x.b + d.b};
}
// the FP64 differences to the left and to the right neighbour, as pairs
__device__ __forceinline__ f2x2 left_difference(d2 x)
{
    const double l = __shfl_up_sync(kAll, x.b, 1);
    return pack(f2_split(x.a - l), f2_split(x.b - x.a));
}
__device__ __forceinline__ f2x2 right_difference(d2 x)
{
    const double r = __shfl_down_sync(kAll, x.a, 1);
    return pack(f2_split(x.b - x.a), f2_split(r - x.b));
}

// The cells of a lane: column of the first, its two (wrapped) columns, and how
// many of the two it writes.  EVEN: nz is even, so that a lane's cells are one
// 16-byte word.
template <bool EVEN>
struct Cells {
    int j, ja, jb, valid;
    __device__ __forceinline__ Cells(int window, int nz)
    {
        const int lane = threadIdx.x & 31;
        j = window * kInner + 2 * (lane - 1);
        valid = lane == 0 || lane == 31 ? 0 : max(0, min(2, nz - j));
        auto wrap = [&](int c) {
            if (c < 0) c += nz;
            return c >= nz ? (c - nz < nz ? c - nz : c % nz) : c;
        };
        ja = wrap(j);
        jb = wrap(j + 1);
    }
    __device__ __forceinline__ d2 load(const double *__restrict__ row) const
    {
        if (EVEN) {
            const double2 v = *reinterpret_cast<const double2 *>(row + ja);
            return d2{v.x, v.y};
        }
        return d2{row[ja], row[jb]};
    }
    // asks L2 for the lane's cells of a row
    __device__ __forceinline__ void prefetch(const double *__restrict__ row) const
    {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(row + ja));
    }
    __device__ __forceinline__ void store(double *__restrict__ row, d2 x) const
    {
        if (EVEN) {
            if (valid) *reinterpret_cast<double2 *>(row + j) = make_double2(x.a, x.b);
        } else {
            if (valid > 0) row[j] = x.a;
            if (valid > 1) row[j + 1] = x.b;
        }
    }
    // the pairs themselves in the doubles' 8 bytes
    __device__ __forceinline__ void store(double *__restrict__ row, f2x2 x) const
    {
        if (EVEN) {
            if (valid)
                *reinterpret_cast<float4 *>(row + j) = make_float4(x.h.x, x.l.x, x.h.y, x.l.y);
        } else {
            float2 *p = reinterpret_cast<float2 *>(row + j);
            if (valid > 0) p[0] = make_float2(x.h.x, x.l.x);
            if (valid > 1) p[1] = make_float2(x.h.y, x.l.y);
        }
    }
};

// The jobs of a grid: windows x chunks of `chunk` rings of `rows`, one per
// warp, window-major so that the warps of a block share ring lines in L1
struct Job {
    int window, i0, i1;
};
__device__ __forceinline__ bool job_of(int nwin, int rows, int chunk, Job &job)
{
    const int k = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const int c = k / nwin;
    job.window = k - c * nwin;
    job.i0 = c * chunk;
    job.i1 = min(job.i0 + chunk, rows);
    return job.i0 < rows;
}

// x < y for a y >= 0, on the integer pipe (a NaN x is not below)
__device__ __forceinline__ bool below(double x, double y)
{
    return __double_as_longlong(x) < __double_as_longlong(y);
}

// x truncated to a float (relative error below 2^-23) for
// 2^-126 <= |x| < 2^128, on the integer pipe; ok is false elsewhere
__device__ __forceinline__ float ftrunc(double x, bool &ok)
{
    const unsigned w1 = (unsigned)__double2hiint(x), w0 = (unsigned)__double2loint(x);
    const unsigned ax = w1 & 0x7fffffffu;
    ok = ax - (897u << 20) < (254u << 20);
    return __uint_as_float(__funnelshift_l(w0, ax - (896u << 20), 3) | (w1 & 0x80000000u));
}

// temperature_floor (floors of Transport, TransportEuler.cpp:122-127, and
// SubStep3): e clamped into [sigma emin_fac, sigma emax_fac], NaN to the lower
// bound, as in the FP64 form.  The FP32 screen passes e only when it lies inside
// the bounds by more than 2^-20 of them (the truncations and roundings of the
// screen are below 2^-22), so an e it passes is one the FP64 clamp leaves alone.
__device__ __forceinline__ double floor_e(double e, double sigma, const Phys &ph)
{
    bool ok_e, ok_s;
    const float ef = ftrunc(e, ok_e), sf = ftrunc(sigma, ok_s);
    const float lo = __fmul_rn(__fmul_rn(sf, ph.emin_fac_f), 1.0f + 0x1p-20f);
    const float hi = __fmul_rn(__fmul_rn(sf, ph.emax_fac_f), 1.0f - 0x1p-20f);
    if (ok_e && ok_s && ef > lo && ef < hi) return e;
    const double emin = sigma * ph.emin_fac;
    const double emax = sigma * ph.emax_fac;
    if (!(e > emin)) e = emin;
    if (!(e < emax)) e = emax;
    return e;
}

}  // namespace win
}  // namespace fgpu
