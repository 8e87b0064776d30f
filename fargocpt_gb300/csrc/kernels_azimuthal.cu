// The FP64 form's azimuthal transport with FARGO orbital advection
// (OneWindTheta, TransportEuler.cpp:270-288) with its arithmetic in float
// pairs (fp64_pair.cuh): QuantitiesAdvection (:292-304: ComputeStarTheta
// :416-466, VanLeerTheta :630-664) with the residual and then the uniform
// velocity.  The ring means and the shift phase (:174-236) come from the
// radial transport's launch (RingPhase); AdvectSHIFT (:238-268) is left to the
// velocity rebuild, which reads each ring's cells at j - its shift.
//
// What bounds it: the FP32 pipe, about 180 operations per transported
// quantity, cell and two passes (1030 instructions per cell; the packed-FP32
// pipe is 72% busy, issue 60%, DRAM 26%).  Everything is arranged around it:
//  * A warp owns a window of 128 consecutive cells of one ring, four per lane
//    in registers, and writes the 120 inner ones.  The four cells at either
//    end are computed along with them: a pass needs two cells on either side,
//    so both passes of a cell follow from the window alone, and no warp waits
//    for another.  (The kernel this replaced kept a ring in shared memory,
//    with two block barriers per quantity and pass: 2470 instructions per cell,
//    issue 53%.)
//  * The neighbours of a lane's first and last cell come by shuffles.  Each
//    cell's difference and limited slope are formed once, and a face's flux
//    once, by the lane that owns the face.
//  * The cells are held as two packed pairs (cells 0, 2 and cells 1, 3 of the
//    lane), so that the left neighbours of the second pack are the first pack
//    itself and the packed FP32 instructions need few register moves.
//  * Both passes of a quantity run back to back: its value between them stays
//    a pair in registers, and the state (sigma, energy) takes one FP64 addition
//    of the two passes' joined increment.  The momenta, which only the velocity
//    rebuild reads, are pairs from the radial pass on.
//  * A window is one job of a flat grid over rings and windows: no block waits
//    for its slowest ring, and the last wave is short (one block per ring with
//    the mean inside: 0.69 ms).
// The output goes to other buffers than the input: the windows of neighbouring
// warps overlap, so an update in place would race.
//
// Measured, ms per pass (ring kernel in shared memory -> this): 2048 x 6144
// 1.377 -> 0.543, 512 x 1536 0.127 -> 0.041, 128 x 384 isothermal 0.020 ->
// 0.010.  At 96 registers (5 blocks per SM, 92 bytes of spills) 0.551.
#include "launch.cuh"
#include "fp64_pair.cuh"
#include "hydro.cuh"
#include "kernels.h"

#include <algorithm>
#include <type_traits>

namespace fgpu {
namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kCells = 4;                              // cells per lane
constexpr int kWindow = 32 * kCells;                   // cells a warp computes
constexpr int kInner = kWindow - 2 * kCells;           // cells it writes

// four consecutive cells of a lane: e holds cells 0 and 2, o cells 1 and 3
struct Quad {
    f2x2 e, o;
};

__device__ __forceinline__ f2 left_of(f2 a)   // the left lane's value
{
    return f2{__shfl_up_sync(kAll, a.h, 1), __shfl_up_sync(kAll, a.l, 1)};
}
__device__ __forceinline__ f2 right_of(f2 a)  // the right lane's value
{
    return f2{__shfl_down_sync(kAll, a.h, 1), __shfl_down_sync(kAll, a.l, 1)};
}

// MC_lim (TransportEuler.cpp:314-323) of two normalised differences
__device__ __forceinline__ f2 mc_limiter(f2 a, f2 b)
{
    auto same = [](f2 x, f2 y) {
        const int ix = __float_as_int(x.h), iy = __float_as_int(y.h);
        return (ix ^ iy) >= 0 && (ix & 0x7fffffff) != 0 && (iy & 0x7fffffff) != 0;
    };
    auto less = [](f2 x, f2 y) {  // |x| < |y|
        const float xh = fabsf(x.h), yh = fabsf(y.h);
        if (xh != yh) return xh < yh;
        return (x.h < 0.f ? -x.l : x.l) < (y.h < 0.f ? -y.l : y.l);
    };
    const f2 zero{0.f, 0.f};
    const f2 mm = same(a, b) ? (less(a, b) ? a : b) : zero;
    const f2 s = f2_sadd(a, b);
    const f2 c{__fmul_rn(0.5f, s.h), __fmul_rn(0.5f, s.l)};
    const f2 d{__fmul_rn(2.0f, mm.h), __fmul_rn(2.0f, mm.l)};
    if (same(c, d)) return less(c, d) ? c : d;
    return zero;
}

// the limited slopes without their constant factor: van Leer's ab / (a + b)
// (its 2 is in the interpolation distance), MC's value as is
template <bool MC>
__device__ __forceinline__ f2x2 limiter(f2x2 a, f2x2 b)
{
    if (MC) return pack(mc_limiter(first(a), first(b)), mc_limiter(second(a), second(b)));
    const f2x2 p = f2_smul(a, b);
    f2x2 r = f2_sdiv(p, f2_sadd(a, b));
    // zero unless a b > 0 (a product that underflows leaves a slope below
    // 2^-63 of the pair format's smallest value)
    const bool x = p.h.x > 0.f, y = p.h.y > 0.f;
    r.h.x = x ? r.h.x : 0.f;
    r.l.x = x ? r.l.x : 0.f;
    r.h.y = y ? r.h.y : 0.f;
    r.l.y = y ? r.l.y : 0.f;
    return r;
}

__device__ __forceinline__ f2 sel(bool c, f2 a, f2 b)
{
    return f2{c ? a.h : b.h, c ? a.l : b.l};
}

// star values at the left faces of a lane's cells: x_u + a s_u from the
// upwind cell u (the left neighbour where pos is set, else the cell itself)
template <bool MC>
__device__ __forceinline__ Quad star(const Quad &X, const Quad &a, bool p0, bool p1, bool p2,
                                     bool p3)
{
    const f2 x3 = left_of(second(X.o));
    const f2x2 left = pack(x3, first(X.o));               // cells -1 and 1
    const f2x2 de = f2_ssub(X.e, left);                   // faces 0 and 2
    const f2x2 dd = f2_ssub(X.o, X.e);                    // faces 1 and 3
    const f2 d4 = right_of(first(de));
    const f2x2 se = limiter<MC>(dd, de);                  // slopes of cells 0 and 2
    const f2x2 so = limiter<MC>(pack(second(de), d4), dd);
    const f2 s3 = left_of(second(so));
    Quad r;
    r.e = f2_sfma(pack(sel(p0, x3, first(X.e)), sel(p2, first(X.o), second(X.e))), a.e,
                  pack(sel(p0, s3, first(se)), sel(p2, first(so), second(se))));
    r.o = f2_sfma(pack(sel(p1, first(X.e), first(X.o)), sel(p3, second(X.e), second(X.o))), a.o,
                  pack(sel(p1, first(se), first(so)), sel(p3, second(se), second(so))));
    return r;
}

// F_j - F_j+1 of a lane's cells
__device__ __forceinline__ Quad divergence(const Quad &F)
{
    const f2 f4 = right_of(first(F.e));
    return Quad{f2_ssub(F.e, F.o), f2_ssub(F.o, pack(second(F.e), f4))};
}

// four consecutive doubles / pairs of a ring; ALIGNED: nz is a multiple of 4,
// so that a lane's cells are one 32-byte sector
template <bool ALIGNED>
__device__ __forceinline__ void load4(const double *__restrict__ p, const int *j, double *x)
{
    if (ALIGNED) {
        const double2 a = *reinterpret_cast<const double2 *>(p + j[0]);
        const double2 b = *reinterpret_cast<const double2 *>(p + j[0] + 2);
        x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
    } else {
#pragma unroll
        for (int k = 0; k < kCells; ++k) x[k] = p[j[k]];
    }
}
template <bool ALIGNED>
__device__ __forceinline__ void store4(double *__restrict__ p, int j, int valid, const double *x)
{
    if (ALIGNED) {
        if (valid > 0) {
            *reinterpret_cast<double2 *>(p + j) = make_double2(x[0], x[1]);
            *reinterpret_cast<double2 *>(p + j + 2) = make_double2(x[2], x[3]);
        }
    } else {
#pragma unroll
        for (int k = 0; k < kCells; ++k)
            if (k < valid) p[j + k] = x[k];
    }
}
// the loaded words as pairs (a pair in the double's 8 bytes, h first)
__device__ __forceinline__ Quad pairs4(const double *x)
{
    f2 p[kCells];
#pragma unroll
    for (int k = 0; k < kCells; ++k)
        p[k] = f2{__int_as_float(__double2loint(x[k])), __int_as_float(__double2hiint(x[k]))};
    return Quad{pack(p[0], p[2]), pack(p[1], p[3])};
}
template <bool ALIGNED>
__device__ __forceinline__ void store4(f2 *__restrict__ p, int j, int valid, const Quad &q)
{
    const f2 x[kCells] = {first(q.e), first(q.o), second(q.e), second(q.o)};
    if (ALIGNED) {
        if (valid > 0) {
            *reinterpret_cast<float4 *>(p + j) = make_float4(x[0].h, x[0].l, x[1].h, x[1].l);
            *reinterpret_cast<float4 *>(p + j + 2) = make_float4(x[2].h, x[2].l, x[3].h, x[3].l);
        }
    } else {
#pragma unroll
        for (int k = 0; k < kCells; ++k)
            if (k < valid) *reinterpret_cast<float2 *>(p + j + k) = make_float2(x[k].h, x[k].l);
    }
}
__device__ __forceinline__ Quad split4(const double *x)
{
    return Quad{pack(f2_split(x[0]), f2_split(x[2])), pack(f2_split(x[1]), f2_split(x[3]))};
}
__device__ __forceinline__ Quad operator+(const Quad &a, const Quad &b)
{
    return Quad{f2_sadd(a.e, b.e), f2_sadd(a.o, b.o)};
}
__device__ __forceinline__ Quad operator*(const Quad &a, const Quad &b)
{
    return Quad{f2_smul(a.e, b.e), f2_smul(a.o, b.o)};
}
__device__ __forceinline__ Quad operator*(const f2x2 &a, const Quad &b)
{
    return Quad{f2_smul(a, b.e), f2_smul(a, b.o)};
}
__device__ __forceinline__ Quad operator/(const Quad &a, const Quad &b)
{
    return Quad{f2_sdiv(a.e, b.e), f2_sdiv(a.o, b.o)};
}
// x += d: the FP64 value plus the joined pair increment
__device__ __forceinline__ void add4(double *x, const Quad &d)
{
    x[0] += f2_to_double(first(d.e));
    x[1] += f2_to_double(first(d.o));
    x[2] += f2_to_double(second(d.e));
    x[3] += f2_to_double(second(d.o));
}

// the quantity rows, chosen by a select chain (an indexed array of pointers
// would sit in local memory)
struct Rows {
    const double *m0, *m1, *m2, *m3, *E, *S;  // the momenta's words are pairs
    f2 *o0, *o1, *o2, *o3;
    double *E_out, *S_out;
    __device__ __forceinline__ const double *in(int q) const
    {
        return q == 0 ? m0 : q == 1 ? m1 : q == 2 ? m2 : q == 3 ? m3 : E;
    }
    __device__ __forceinline__ f2 *out(int q) const
    {
        return q == 0 ? o0 : q == 1 ? o1 : q == 2 ? o2 : o3;
    }
};

constexpr int kThreads = 128;

template <bool ADIABATIC, bool ALIGNED, bool MC>
__global__ void __launch_bounds__(kThreads, 4)
    k_transport_azimuthal_p(int nz, int nr, int windows, int fast,
                            const double *__restrict__ vaz, Rows rows,
                            const RingPhase *__restrict__ phase)
{
    follow_predecessor();
    const int lane = threadIdx.x & 31;
    const int job = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const int i = job / windows;
    if (i >= nr) return;
    const int c0 = (job - i * windows) * kInner;
    const size_t row = (size_t)i * nz;
    vaz += row;
    const RingPhase &ring = phase[i];
    {
        const int base = c0 + (lane - 1) * kCells;
        // cells this lane writes: whole ones of the window's inner 120
        const int valid = lane == 0 || lane == 31 ? 0 : min(kCells, nz - base);
        int j[kCells];
#pragma unroll
        for (int k = 0; k < kCells; ++k) {
            int b = base + k;
            if (b < 0) b += nz;
            if (b >= nz) b = b - nz < nz ? b - nz : b % nz;
            j[k] = b;
        }
        double v[kCells], s[kCells], next[kCells];
        load4<ALIGNED>(vaz, j, v);
        load4<ALIGNED>(rows.S + row, j, s);
        load4<ALIGNED>(rows.in(0) + row, j, next);
        // the other rows come from DRAM: ask L2 for them now
#pragma unroll
        for (int q = 1; q < (ADIABATIC ? 5 : 4); ++q)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(rows.in(q) + row + j[0]));
        const double about = ring.about;
        const f2x2 au = pack(f2{ring.au.x, ring.au.y});
        const bool pu = ring.upwind;
        const f2 dxp{MC ? 0.5f : 1.0f, 0.f}, dxn = f2_neg(dxp);
        // the residual velocity times k dt, the upwind sides and distances
#pragma unroll
        for (int k = 0; k < kCells; ++k) v[k] -= about;
        const Quad vk = pack(f2{ring.kdt.x, ring.kdt.y}) * split4(v);
        const bool p0 = vk.e.h.x > 0.f, p1 = vk.o.h.x > 0.f, p2 = vk.e.h.y > 0.f,
                   p3 = vk.o.h.y > 0.f;
        const Quad a{f2_ssub(pack(sel(p0, dxp, dxn), sel(p2, dxp, dxn)), vk.e),
                     f2_ssub(pack(sel(p1, dxp, dxn), sel(p3, dxp, dxn)), vk.o)};
        // DensityStar and the factor dxrad S* v / Surf every flux shares
        const Quad S = split4(s);
        const Quad c = (pack(f2{ring.face.x, ring.face.y}) * vk) * star<MC>(S, a, p0, p1, p2, p3);
        Quad ds = divergence(c);
        const Quad S1 = S + ds;
        Quad cu = c;
        if (fast) {
            cu = pack(f2{ring.fu.x, ring.fu.y}) * star<MC>(S1, Quad{au, au}, pu, pu, pu, pu);
            ds = ds + divergence(cu);
        }
        add4(s, ds);
        store4<ALIGNED>(rows.S_out + row, base, valid, s);

#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
            const Quad Q = pairs4(next);
            if (q < 3 || ADIABATIC) load4<ALIGNED>(rows.in(q + 1) + row, j, next);
            Quad d = divergence(star<MC>(Q / S, a, p0, p1, p2, p3) * c);
            if (fast)
                d = d + divergence(star<MC>((Q + d) / S1, Quad{au, au}, pu, pu, pu, pu) * cu);
            // one rounding of the momentum for the two passes
            store4<ALIGNED>(rows.out(q) + row, base, valid, Q + d);
        }
        if (ADIABATIC) {
            const Quad Q = split4(next);
            Quad d = divergence(star<MC>(Q / S, a, p0, p1, p2, p3) * c);
            if (fast)
                d = d + divergence(star<MC>((Q + d) / S1, Quad{au, au}, pu, pu, pu, pu) * cu);
            add4(next, d);
            store4<ALIGNED>(rows.E_out + row, base, valid, next);
        }
    }
}

}  // namespace

void launch_transport_azimuthal_pair(const Launch &L, double *const mom[4], const double *E,
                                     const double *S, const double *vaz,
                                     double *const mom_out[4], double *E_out, double *S_out,
                                     const RingPhase *phase)
{
    auto out = [&](int q) { return reinterpret_cast<f2 *>(mom_out[q]); };
    const Rows r{mom[0], mom[1], mom[2], mom[3], E,     S,
                 out(0), out(1), out(2), out(3), E_out, S_out};
    const int windows = (L.g.nz + kInner - 1) / kInner, per = kThreads / 32;
    const bool aligned = L.g.nz % kCells == 0;
    auto pick = [&](auto adi, auto al) {
        return L.ph.limiter_mc ? k_transport_azimuthal_p<adi.value, al.value, true>
                               : k_transport_azimuthal_p<adi.value, al.value, false>;
    };
    using T = std::true_type;
    using F = std::false_type;
    auto k = L.ph.adiabatic ? (aligned ? pick(T{}, T{}) : pick(T{}, F{}))
                            : (aligned ? pick(F{}, T{}) : pick(F{}, F{}));
    launch(k, (L.g.nr * windows + per - 1) / per, kThreads, 0, L.stream,
        L.g.nz, L.g.nr, windows, L.ph.fast_transport, vaz, r, phase);
}

}  // namespace fgpu
