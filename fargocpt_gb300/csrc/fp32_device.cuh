// Device bodies of the FP32-mixed hydro step, shared by the single-disk
// kernels (kernels_fp32.cu) and the batched many-disk kernels
// (batch_fp32.cu).  Each body updates one cell, one column or one ring of one
// disk; the kernels around them only decide which disk, ring and column a
// thread works on.  The storage conventions (residual v_phi about v_K(Rmed),
// potential residual about -G M / Rmed, compensated sigma hi + lo) are
// described at the top of kernels_fp32.cu.
#pragma once

#include "fp32_engine.h"

#include <cuda_runtime.h>

namespace fgpu32 {

#define CELL(i, j) ((size_t)(i) * (size_t)nz + (size_t)(j))

__device__ __forceinline__ int jnext(int j, int nz) { return j == nz - 1 ? 0 : j + 1; }
__device__ __forceinline__ int jprev(int j, int nz) { return j == 0 ? nz - 1 : j - 1; }

__device__ __forceinline__ float lim_f(float a, float b, int mc)
{
    if (mc) {
        float mm = 0.f;
        if (a * b > 0.f) mm = fabsf(a) < fabsf(b) ? a : b;
        const float c = 0.5f * (a + b), d = 2.f * mm;
        if (c * d > 0.f) return fabsf(c) < fabsf(d) ? c : d;
        return 0.f;
    }
    if (a * b > 0.f) return __fdividef(2.f * a * b, a + b);
    return 0.f;
}

// hi + lo + inc as a compensated pair: y = lo + inc is small next to hi, so
// Fast2Sum (Dekker 1971) recovers the rounding error of hi + y exactly.
__device__ __forceinline__ void comp_add(float &hi, float &lo, float inc)
{
    const float y = lo + inc;
    const float s = hi + y;
    lo = y - (s - hi);
    hi = s;
}

// The star values and fluxes of the azimuthal passes with the rounding of
// every operation fixed (an explicit FMA where the value is interpolated),
// so that the strided and the register-blocked ring kernels, whose code the
// compiler would otherwise contract differently, give the same bits; the
// passes spell out the specific values (q / sigma as q times 1 / sigma) and
// the slopes' differences and scaling for the same reason (the blocked kernel
// holds a specific value in a register where it is differenced, the strided
// one reloads it from shared memory, and only the former may fuse the two).
//   upwind value on the positive side: W_jm + (dx - ksi) D_jm
//   on the negative side:              W_j  - (dx + ksi) D_j
__device__ __forceinline__ float star_pos(float w, float d, float dx, float ksi)
{
    return __fmaf_rn(__fsub_rn(dx, ksi), d, w);
}
__device__ __forceinline__ float star_neg(float w, float d, float dx, float ksi)
{
    return __fmaf_rn(-__fadd_rn(dx, ksi), d, w);
}
// X_u + a D_u and the neighbour difference (X_u - X_u1) + a (D_u - D_u1)
__device__ __forceinline__ float star_at(float x, float d, float a) { return __fmaf_rn(a, d, x); }
__device__ __forceinline__ float star_diff(float xu, float xu1, float du, float du1, float a)
{
    return __fmaf_rn(a, __fsub_rn(du, du1), __fsub_rn(xu, xu1));
}
// q += c (qs dS* + S*_{j+1} dq*) of the uniform pass
__device__ __forceinline__ float uniform_update(float q, float c, float qs, float dss, float fs,
                                                float dqs)
{
    return __fadd_rn(q, __fmul_rn(c, __fmaf_rn(qs, dss, __fmul_rn(fs, dqs))));
}

__device__ __forceinline__ float tfloor(float e, float sigma, const PhysF &ph)
{
    const float emin = sigma * ph.emin_fac;
    const float emax = sigma * ph.emax_fac;
    if (!(e > emin)) e = emin;
    if (!(e < emax)) e = emax;
    return e;
}

__device__ __forceinline__ double warp_sum_d(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_min_f(float v)
{
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}
template <typename T, T (*WARP)(T)>
__device__ __forceinline__ T block_reduce(T v, T *red, T neutral)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nw = (blockDim.x + 31) >> 5;
    v = WARP(v);
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    if (wid == 0) {
        T x = lane < nw ? red[lane] : neutral;
        x = WARP(x);
        if (lane == 0) red[32] = x;
    }
    __syncthreads();
    return red[32];
}
__device__ __forceinline__ double bsum_d(double v, double *red)
{
    return block_reduce<double, warp_sum_d>(v, red, 0.0);
}
__device__ __forceinline__ float bmin_f(float v, float *red)
{
    return block_reduce<float, warp_min_f>(v, red, 3.0e38f);
}

__device__ __forceinline__ float warp_max_f(float v)
{
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ long long warp_sum_ll(long long v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Ring sums that do not depend on the block's shape.  Every value is rounded
// to a multiple of 2^-k and the resulting 64-bit integers are added; integer
// addition is associative, so neither the tile shape a kernel runs with nor
// the order of the threads changes a bit of the result.  k is the largest
// exponent for which n values of at most the block's largest |x| stay below
// 2^62 in total; the sum is then within n 2^-k (about 2^-51 n max|x|) of the
// exact one.  Every thread of the block must call both steps.
//
// Step 1: the scale, from the block's largest |x| (an exact reduction).
__device__ __forceinline__ int exact_sum_scale(float local_absmax, int n, float *redf)
{
    const float m = block_reduce<float, warp_max_f>(local_absmax, redf, 0.f);
    int e = 0;
    frexpf(m, &e);                // m < 2^e
    const int ln = 32 - __clz(n);  // n < 2^ln
    return 62 - e - ln;
}
// (x 2^k in two exact multiplications: |x 2^k| < 2^62, and what a first step
// towards zero rounds in the subnormals is far below 1/2)
__device__ __forceinline__ long long to_fixed(float x, int k)
{
    const int k1 = k >> 1;
    const float a = __int_as_float((127 + k1) << 23), b = __int_as_float((127 + (k - k1)) << 23);
    return __float2ll_rn(__fmul_rn(__fmul_rn(x, a), b));
}
// Step 2: the sum of the threads' integer partial sums.
__device__ __forceinline__ double exact_sum_result(long long part, int k, long long *redl)
{
    const long long s = block_reduce<long long, warp_sum_ll>(part, redl, 0LL);
    return ldexp((double)s, -k);
}

// Mean of row[0 .. n-1] (global memory, shared by the block; the last division
// by one thread, red[32] to the others).
__device__ __forceinline__ float exact_row_mean(const float *row, int n, float *redf,
                                                long long *redl)
{
    const int bs = blockDim.x, tid = threadIdx.x;
    float m = 0.f;
#pragma unroll 8
    for (int j = tid; j < n; j += bs) m = fmaxf(m, fabsf(row[j]));
    const int k = exact_sum_scale(m, n, redf);
    long long part = 0;
#pragma unroll 8
    for (int j = tid; j < n; j += bs) part += to_fixed(row[j], k);
    const long long s = block_reduce<long long, warp_sum_ll>(part, redl, 0LL);
    if (tid == 0) redf[32] = (float)(ldexp((double)s, -k) / (double)n);
    __syncthreads();
    return redf[32];
}

// ---------------------------------------------------------------------------
// Four cells of a ring per thread, for the kernels that form cells one by one.
// Such a cell is 20 to 60 operations on some ten loaded values; with one cell per
// thread the index arithmetic, the ring's table values, the ring search of the
// batch and the launch's prologue were most of the 240 to 330 instructions it
// took (issue bound them, at a third of the memory's rate).  2048 x 6144 cells,
// one cell -> four: potential 0.102 -> 0.047 ms, source terms 0.102 -> 0.059,
// artificial pressures 0.102 -> 0.047, their update 0.110 -> 0.079, stress 0.102
// -> 0.061, viscous update 0.215 -> 0.122, finish 0.134 -> 0.087 (now near the
// memory's rate: 7 to 14 rows of 4 bytes each); a batch of 16 disks, 4.8M
// cells: 0.53 -> 0.30 ms together.
// VEC (nz a multiple of 4): adjacent cells in 16-byte accesses, whose neighbours
// within the four come from registers.  Otherwise rows do not start on 16-byte
// boundaries: cells `stride` apart in scalar accesses (adjacent ones would spread
// each access over four times the cache lines); those past the ring's end repeat
// its last cell and are not stored.
// ---------------------------------------------------------------------------
template <bool VEC>
struct Quad {
    int nz, first, stride;

    __device__ __forceinline__ int col(int k) const
    {
        return VEC ? first + k : min(first + k * stride, nz - 1);
    }
    __device__ __forceinline__ void load(const float *p, size_t row, float (&x)[4]) const
    {
        if (VEC) {
            const float4 v = *reinterpret_cast<const float4 *>(p + row + first);
            x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) x[k] = p[row + col(k)];
        }
    }
    // the left (right) neighbours of the cells x
    __device__ __forceinline__ void left(const float *p, size_t row, const float (&x)[4],
                                         float (&l)[4]) const
    {
        if (VEC) {
            l[0] = p[row + jprev(first, nz)];
            l[1] = x[0], l[2] = x[1], l[3] = x[2];
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) l[k] = p[row + jprev(col(k), nz)];
        }
    }
    __device__ __forceinline__ void right(const float *p, size_t row, const float (&x)[4],
                                          float (&r)[4]) const
    {
        if (VEC) {
            r[0] = x[1], r[1] = x[2], r[2] = x[3];
            r[3] = p[row + jnext(first + 3, nz)];
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) r[k] = p[row + jnext(col(k), nz)];
        }
    }
    __device__ __forceinline__ void store(float *p, size_t row, const float (&x)[4]) const
    {
        if (VEC) {
            *reinterpret_cast<float4 *>(p + row + first) = make_float4(x[0], x[1], x[2], x[3]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (first + k * stride < nz) p[row + first + k * stride] = x[k];
        }
    }
};
#define QUAD for (int k = 0; k < 4; ++k)

// ---------------------------------------------------------------------------
// Potential residual Phi - Phi_K (CalculateNbodyPotential, Pframeforce.cpp:21-86)
// ---------------------------------------------------------------------------
// Klahr's u^4 - 2 u^3 + 2 u inside r_sm (u the distance in it)
__device__ __forceinline__ float klahr_factor(float u)
{
    return fmaf(__fmul_rn(__fmul_rn(u, u), u), u, -__fmul_rn(__fmul_rn(2.f * u, u), u)) + 2.f * u;
}

// (fused multiply-adds of these substeps are spelled out where the compiler
// would have a choice, so that every kernel built from them rounds alike)
template <class Q>
__device__ __forceinline__ void potential_cells(
    const Q &q, const GeoF &g, const TablesF &t, const PhysF &ph, const BodiesF &b,
    const float *__restrict__ H, float *__restrict__ pot, int i)
{
    const size_t row = (size_t)i * g.nz;
    // the cell centres as float pairs (x = xh + xl): the product's rounding
    // error by FMA plus the cross terms of the split factors; the distance to
    // a body then loses nothing to cancellation however close the body is
    const float rh = t.Rmed[i], rl = t.RmedLo[i];
    float h[4], ch[4], cl[4], sh[4], sl[4], xh[4], yh[4], xl[4], yl[4], s2[4], acc[4];
    q.load(H, row, h);
    q.load(t.cosHi, 0, ch);
    q.load(t.cosLo, 0, cl);
    q.load(t.sinHi, 0, sh);
    q.load(t.sinLo, 0, sl);
#pragma unroll
    QUAD {
        xh[k] = rh * ch[k], yh[k] = rh * sh[k];
        xl[k] = fmaf(rh, ch[k], -xh[k]) + fmaf(rh, cl[k], rl * ch[k]);
        yl[k] = fmaf(rh, sh[k], -yh[k]) + fmaf(rh, sl[k], rl * sh[k]);
        const float eps = ph.eps_smooth * h[k];
        s2[k] = eps * eps;
        acc[k] = 0.f;
    }
    for (int n = 0; n < b.n; ++n) {
        if (n == 0 && b.star_at_origin) {
            // -G M / sqrt(r^2 + eps^2) + G M / r without cancellation:
            // 1/r - 1/d = (d - r) / (r d) = eps^2 / ((d + r) r d)
            const float gm = b.gm[0];
#pragma unroll
            QUAD {
                const float d = sqrtf(rh * rh + s2[k]);
                acc[k] += gm * s2[k] / ((d + rh) * rh * d);
            }
        } else if (n == 0) {
            // central object off the origin: residual against -G M / r in FP64
            const double rmed = t.Rmed_d[i], inv = t.InvRmed_d[i];
#pragma unroll
            QUAD {
                const double xd = rmed * t.cos_d[q.col(k)], yd = rmed * t.sin_d[q.col(k)];
                const double dx = xd - b.x[0], dy = yd - b.y[0];
                const float d2 = (float)(dx * dx + dy * dy) + s2[k];
                const float inv_d = rsqrtf(d2);
                float fk = 1.f;
                if (b.rsm[0] > 0.f) {
                    const float dsm = d2 * inv_d;
                    if (dsm < b.rsm[0]) fk = klahr_factor(dsm / b.rsm[0]);
                }
                acc[k] += (float)(-(double)b.gm[0] * fk / sqrt(dx * dx + dy * dy + (double)s2[k]) +
                                  (double)b.gm_ref * inv);
            }
        } else {
            const float bxh = b.xh[n], bxl = b.xl[n], byh = b.yh[n], byl = b.yl[n];
            const float mgm = -b.gm[n], rsm = b.rsm[n];
#pragma unroll
            QUAD {
                const float dx = (xh[k] - bxh) + (xl[k] - bxl);
                const float dy = (yh[k] - byh) + (yl[k] - byl);
                const float d2 = fmaf(dx, dx, fmaf(dy, dy, s2[k]));
                const float inv_d = rsqrtf(d2);
                float fk = 1.f;
                if (rsm > 0.f) {
                    const float dsm = d2 * inv_d;
                    if (dsm < rsm) fk = klahr_factor(dsm / rsm);
                }
                acc[k] = fmaf(__fmul_rn(mgm, inv_d), fk, acc[k]);
            }
        }
    }
#pragma unroll
    QUAD acc[k] = fmaf(-b.iy, yh[k] + yl[k], fmaf(-b.ix, xh[k] + xl[k], acc[k]));
    q.store(pot, row, acc);
}

// ---------------------------------------------------------------------------
// momentum sources (SourceEuler.cpp:325-428) in residual form; rows 0..nr
// ---------------------------------------------------------------------------
template <class Q>
__device__ __forceinline__ void source_cells(
    const Q &q, const GeoF &g, const TablesF &t, float dt, const float *__restrict__ S,
    const float *__restrict__ P, const float *__restrict__ pot,
    const float *__restrict__ vr_in, const float *__restrict__ dv_in,
    float *__restrict__ vr_out, float *__restrict__ dv_out, int i)
{
    const int nz = g.nz, nr = g.nr;
    const size_t row = (size_t)i * nz, below = row - nz;
    float vr[4], v[4], p[4], s[4], ph[4];
    q.load(vr_in, row, vr);
    const bool active = i >= 1 && i < nr - 1;
    if (i < nr) q.load(dv_in, row, v);
    if (active) {
        q.load(P, row, p);
        q.load(S, row, s);
        q.load(pot, row, ph);
    }
    if (i >= 2 && active) {
        const float invdr = t.InvDiffRmed[i], kbal = t.Kbal[i], aface = t.Aface[i],
                    invr = t.InvRinf[i], off = t.RinfOff[i];
        float pm[4], sm[4], phm[4], vn[4], vb[4], vbn[4];
        q.load(P, below, pm);
        q.load(S, below, sm);
        q.load(pot, below, phm);
        q.load(dv_in, below, vb);
        q.right(dv_in, row, v, vn);
        q.right(dv_in, below, vb, vbn);
#pragma unroll
        QUAD {
            const float gradp = 2.f * __fdividef(p[k] - pm[k], s[k] + sm[k]) * invdr;
            const float gradphi = (ph[k] - phm[k]) * invdr;
            float d = 0.25f * (v[k] + vn[k] + vb[k] + vbn[k]);
            // in a rotating frame the reference's vt (frame velocities averaged,
            // plus Rinf OmegaFrame; SourceEuler.cpp:355-364) is the inertial mean
            // plus OmegaFrame (Rinf - the mean of the two Rmed)
            if (g.omega_f != 0.f) d += g.omega_f * off;
            // vt^2 / r - dPhi_K/dr = Kbal + (2 A d + d^2) / Rinf
            const float centri = kbal + (2.f * aface + d) * d * invr;
            vr[k] += dt * (-gradp - gradphi + centri);
        }
    }
    q.store(vr_out, row, vr);
    if (i < nr) {
        if (active) {
            const float invdx = t.InvDxSrc[i];
            float pl[4], sl[4], phl[4];
            q.left(P, row, p, pl);
            q.left(S, row, s, sl);
            q.left(pot, row, ph, phl);
#pragma unroll
            QUAD {
                const float gradp = 2.f * __fdividef(p[k] - pl[k], s[k] + sl[k]) * invdx;
                const float gradphi = (ph[k] - phl[k]) * invdx;
                v[k] = v[k] + dt * (-gradp - gradphi);
            }
        }
        q.store(dv_out, row, v);
    }
}

// div v, (vr1 Rinf[i+1] - vr0 Rinf[i]) / ((Rsup - Rinf) Rmed) + dv_phi / (dphi
// Rmed), regrouped exactly (Rinf[i+1] = Rsup[i]) so that no product cancels; the
// fused form is spelled out so that every kernel rounds it the same way
__device__ __forceinline__ float div_v_of(float vr0, float vr1, float dvp, float invdphi,
                                          float rsupidrr, float invrmed)
{
    return fmaf(__fmul_rn(dvp, invdphi), invrmed,
                fmaf(vr1 - vr0, rsupidrr, __fmul_rn(vr0, invrmed)));
}

// compression heating + SN q and energy update + T floor
template <class Q>
__device__ __forceinline__ void artvisc_q_cells(
    const Q &q, const GeoF &g, const TablesF &t, const PhysF &ph, float dt,
    const float *__restrict__ S, const float *__restrict__ vr, const float *__restrict__ dv,
    float *__restrict__ E, float *__restrict__ Qr, float *__restrict__ Qp, int i)
{
    const int nz = g.nz, nr = g.nr;
    const size_t row = (size_t)i * nz;
    float vr0[4], vr1[4], d0[4], dvp[4], sig[4], e[4] = {};
    q.load(vr, row, vr0);
    q.load(vr, row + nz, vr1);
    q.load(dv, row, d0);
    q.right(dv, row, d0, dvp);
    q.load(S, row, sig);
    if (ph.adiabatic) q.load(E, row, e);
    const float rsupidrr = t.RsupIDRR[i], invrmed = t.InvRmed[i], invdrsup = t.InvDiffRsup[i],
                invdxt = t.InvDxTheta[i], lsq = t.LSqTW[i];
    const bool active = i >= 1 && i < nr - 1;
#pragma unroll
    QUAD dvp[k] = dvp[k] - d0[k];
    if (ph.adiabatic && i < nr - 1) {
#pragma unroll
        QUAD {
            const float div_v = div_v_of(vr0[k], vr1[k], dvp[k], g.invdphi, rsupidrr, invrmed);
            e[k] = e[k] * __expf(-ph.gm1 * dt * div_v);
        }
    }
    if (ph.art_visc_sn) {
        float qr[4], qp[4];
#pragma unroll
        QUAD {
            const float dv_r = vr1[k] - vr0[k];
            qr[k] = dv_r < 0.f ? ph.C2 * sig[k] * (dv_r * dv_r) : 0.f;
            qp[k] = dvp[k] < 0.f ? ph.C2 * sig[k] * (dvp[k] * dvp[k]) : 0.f;
            if (ph.adiabatic && ph.dissipation && active)
                e[k] = e[k] - dt * qr[k] * dv_r * invdrsup - dt * qp[k] * dvp[k] * invdxt;
        }
        q.store(Qr, row, qr);
        q.store(Qp, row, qp);
    }
    if (ph.art_visc_tw) {
        // update_with_artificial_viscosity_TW, artificial_viscosity.cpp:52-91
        // (velocity differences within a ring are the same for the residual)
        float qr[4], qp[4];
#pragma unroll
        QUAD {
            const float eps_rr = __fmul_rn(vr1[k] - vr0[k], invdrsup);
            const float eps_pp = __fmul_rn(
                invrmed, __fadd_rn(__fmul_rn(dvp[k], g.invdphi), 0.5f * (vr1[k] + vr0[k])));
            const float div_V = fminf(__fadd_rn(eps_rr, eps_pp), 0.f);
            const float lsig = lsq * sig[k];
            qr[k] = lsig * -div_V * fmaf(-(1.f / 3.f), div_V, eps_rr);
            qp[k] = lsig * -div_V * fmaf(-(1.f / 3.f), div_V, eps_pp);
            if (ph.adiabatic && ph.dissipation && active) {
                const float d = __fsub_rn(eps_rr, eps_pp);
                const float squares = fmaf(d, d, fmaf(eps_rr, eps_rr, __fmul_rn(eps_pp, eps_pp)));
                e[k] = fmaf(-lsig * div_V * (1.f / 3.f) * squares, dt, e[k]);
            }
        }
        q.store(Qr, row, qr);
        q.store(Qp, row, qp);
    }
    if (ph.adiabatic) {
        if (ph.dissipation) {
#pragma unroll
            QUAD e[k] = tfloor(e[k], sig[k], ph);
        }
        q.store(E, row, e);
    }
}

template <class Q>
__device__ __forceinline__ void artvisc_v_cells(
    const Q &q, const GeoF &g, const TablesF &t, const PhysF &ph, float dt,
    const float *__restrict__ S, const float *__restrict__ E, const float *__restrict__ Qr,
    const float *__restrict__ Qp, float *__restrict__ vr, float *__restrict__ dv,
    float *__restrict__ cs, float *__restrict__ H, float *__restrict__ nu, int i)
{
    const int nz = g.nz, nr = g.nr;
    const size_t row = (size_t)i * nz, below = row - nz;
    float s[4];
    q.load(S, row, s);
    const bool radial = i >= 2 && i < nr - 1, azimuthal = i >= 1 && i < nr - 1;
    if (azimuthal && (ph.art_visc_sn || ph.art_visc_tw)) {
        float sl[4], sb[4], qr[4], qrb[4], qp[4], qpl[4], qpb[4], v[4], d[4];
        q.load(Qp, row, qp);
        q.left(Qp, row, qp, qpl);
        q.left(S, row, s, sl);
        q.load(dv, row, d);
        if (radial) {
            q.load(S, below, sb);
            q.load(Qr, row, qr);
            q.load(Qr, below, qrb);
            q.load(vr, row, v);
            if (ph.art_visc_tw) q.load(Qp, below, qpb);
        }
        if (ph.art_visc_sn) {
            const float invdr = t.InvDiffRmed[i], invdxt = t.InvDxTheta[i];
            if (radial) {
#pragma unroll
                QUAD v[k] -= dt * 2.f * __fdividef(qr[k] - qrb[k], s[k] + sb[k]) * invdr;
            }
#pragma unroll
            QUAD d[k] -= dt * 2.f * __fdividef(qp[k] - qpl[k], s[k] + sl[k]) * invdxt;
        }
        if (ph.art_visc_tw) {
            // artificial_viscosity.cpp:93-139
            const float invdx = t.InvDxSrc[i];
#pragma unroll
            QUAD d[k] += __fdividef(dt, 0.5f * (s[k] + sl[k])) * invdx * (qp[k] - qpl[k]);
            if (radial) {
                const float two = t.TwoOverDRmed2[i], r0 = t.Rmed[i], rb = t.Rmed[i - 1],
                            dr = t.DRmed[i];
#pragma unroll
                QUAD {
                    const float fac = ph.rvf * __fdividef(dt, 0.5f * (s[k] + sb[k])) * two;
                    const float rhs = fmaf(-(0.5f * (qp[k] + qpb[k])), dr,
                                           fmaf(qr[k], r0, -__fmul_rn(qrb[k], rb)));
                    v[k] = fmaf(fac, rhs, v[k]);
                }
            }
        }
        if (radial) q.store(vr, row, v);
        q.store(dv, row, d);
    }
    if (ph.adiabatic) {
        float e[4], c[4], h[4], n[4];
        q.load(E, row, e);
        const float hfac = t.HFacAdi[i];
#pragma unroll
        QUAD {
            c[k] = sqrtf(ph.g_gm1 * __fdividef(e[k], s[k]));
            h[k] = c[k] * hfac;
            n[k] = ph.alpha > 0.f ? ph.alpha * h[k] * c[k] : ph.constant_viscosity;
        }
        q.store(cs, row, c);
        q.store(H, row, h);
        q.store(nu, row, n);
    }
}

// stress tensor (viscosity.cpp:139-254); tau_r_phi adds the Keplerian shear
template <class Q>
__device__ __forceinline__ void stress_cells(
    const Q &q, const GeoF &g, const TablesF &t, const float *__restrict__ S,
    const float *__restrict__ vr, const float *__restrict__ dv, const float *__restrict__ nu,
    float *__restrict__ divv, float *__restrict__ trr, float *__restrict__ tpp,
    float *__restrict__ trp, int i)
{
    const int nz = g.nz;
    const size_t row = (size_t)i * nz, below = row - nz;
    float vr0[4], vr1[4], d0[4], dvp[4], n[4], sg[4], x[4], y[4], z[4];
    q.load(vr, row, vr0);
    q.load(vr, row + nz, vr1);
    q.load(dv, row, d0);
    q.right(dv, row, d0, dvp);
    q.load(nu, row, n);
    q.load(S, row, sg);
    const float rsupidrr = t.RsupIDRR[i], invrmed = t.InvRmed[i], invdrsup = t.InvDiffRsup[i];
#pragma unroll
    QUAD {
        dvp[k] = dvp[k] - d0[k];
        const float d = div_v_of(vr0[k], vr1[k], dvp[k], g.invdphi, rsupidrr, invrmed);
        x[k] = d;
        const float drr = (vr1[k] - vr0[k]) * invdrsup;
        y[k] = 2.f * n[k] * sg[k] * (drr - (1.f / 3.f) * d);
        const float dpp = fmaf(__fmul_rn(dvp[k], g.invdphi), invrmed,
                               __fmul_rn(0.5f * (vr1[k] + vr0[k]), invrmed));
        z[k] = 2.f * n[k] * sg[k] * (dpp - (1.f / 3.f) * d);
    }
    q.store(divv, row, x);
    q.store(trr, row, y);
    q.store(tpp, row, z);
    if (i >= 1) {
        float db[4], vl[4], nb[4], nl[4], nbl[4], sb[4], sl[4], sbl[4];
        q.load(dv, below, db);
        q.left(vr, row, vr0, vl);
        q.load(nu, below, nb);
        q.left(nu, row, n, nl);
        q.left(nu, below, nb, nbl);
        q.load(S, below, sb);
        q.left(S, row, sg, sl);
        q.left(S, below, sb, sbl);
        const float shear = t.Shear[i], invrb = t.InvRmed[i - 1], invdr = t.InvDiffRmed[i],
                    rinf = t.Rinf[i], invrinf = t.InvRinf[i];
#pragma unroll
        QUAD {
            const float dvazirdr = shear + (d0[k] * invrmed - db[k] * invrb) * invdr;
            const float dvrdphi = (vr0[k] - vl[k]) * g.invdphi;
            const float drp = rinf * dvazirdr + dvrdphi * invrinf;
            const float n4 = 0.25f * (n[k] + nb[k] + nl[k] + nbl[k]);
            const float s4 = 0.25f * (sg[k] + sb[k] + sl[k] + sbl[k]);
            x[k] = n4 * s4 * drp;
        }
        q.store(trp, row, x);
    }
}

// StabilizeViscosity's correction factors (viscosity.cpp:256-348), rows
// 1 .. nr - 1, from nu and sigma (nu sigma at the centres, the four-cell
// averages at the r-phi corners; row nr of the latter is zero)
__device__ __forceinline__ float nusig_rp_f(const float *nu, const float *S, int nz, int i, int j)
{
    const int jp = jprev(j, nz);
    const float n = 0.25f * (nu[CELL(i, j)] + nu[CELL(i - 1, j)] + nu[CELL(i, jp)] +
                             nu[CELL(i - 1, jp)]);
    const float s = 0.25f * (S[CELL(i, j)] + S[CELL(i - 1, j)] + S[CELL(i, jp)] +
                             S[CELL(i - 1, jp)]);
    return n * s;
}

__device__ __forceinline__ void visc_corr_cell(const GeoF &g, const TablesF &t,
                                               const float *__restrict__ S,
                                               const float *__restrict__ nu,
                                               float *__restrict__ corr_phi,
                                               float *__restrict__ corr_r, int i, int j)
{
    const int nz = g.nz, nr = g.nr;
    const size_t c = CELL(i, j);
    const int jp = jprev(j, nz), jn = jnext(j, nz);
    const float rp = nusig_rp_f(nu, S, nz, i, j);
    const float rp_ip = i + 1 < nr ? nusig_rp_f(nu, S, nz, i + 1, j) : 0.f;
    const float rp_jp = nusig_rp_f(nu, S, nz, i, jn);
    const float ns = nu[c] * S[c];
    const float ns_jm = nu[CELL(i, jp)] * S[CELL(i, jp)];
    const float ns_im = nu[CELL(i - 1, j)] * S[CELL(i - 1, j)];
    const float cphi_rp = -t.InvRmed[i] * t.TwoOverDRa2[i] *
                          (rp_ip * t.Ra3IDRmed[i + 1] + rp * t.Ra3IDRmed[i]);
    const float cphi_pp = -t.F43[i] * (ns + ns_jm);
    corr_phi[c] = (cphi_rp + cphi_pp) / (0.5f * (S[c] + S[CELL(i, jp)]) * t.Rmed[i]);
    const float cr_rp = -(rp_jp + rp) * t.CrRp[i];
    const float cr_pp = -0.5f * (ns * t.CrPp1[i] + ns_im * t.CrPp2[i]);
    const float cr_rr = t.InvDiffRmed[i] * (ns * t.CrRr1[i] + ns_im * t.CrRr2[i]);
    corr_r[c] = t.CrScale[i] * (cr_rr + cr_rp + cr_pp) / (0.5f * (S[c] + S[CELL(i - 1, j)]));
}

// viscous velocity update + SubStep3.  mode bits: 1 velocities
// (viscosity.cpp:355-421), 2 heating/cooling rates, 4 energy update
// (SourceEuler.cpp:859-954)
template <class Q>
__device__ __forceinline__ void viscous_cells(
     const Q &q, const GeoF &g, const TablesF &t, const PhysF &ph, float dt, float beta_inv,
    int mode, const float *__restrict__ S, const float *__restrict__ trr,
    const float *__restrict__ tpp, const float *__restrict__ trp,
    const float *__restrict__ divv, const float *__restrict__ nu, const float *__restrict__ H,
    const float *__restrict__ S0, const float *__restrict__ E0, float *__restrict__ vr,
    float *__restrict__ dv, float *__restrict__ E, float *__restrict__ qplus,
    float *__restrict__ qminus, const float *__restrict__ corr_phi,
    const float *__restrict__ corr_r, int i)
{
    const int nz = g.nz, nr = g.nr;
    const size_t row = (size_t)i * nz, below = row - nz, above = row + nz;
    const bool active = i >= 1 && i < nr - 1;
    // pseudo-implicit limiter of StabilizeViscosity 1, viscosity.cpp:395-399
    auto stabilized = [&](float d, float cc) {
        const float a = 1.f + dt * cc;
        return d * (1.f / (fmaxf(a, 0.f) - dt * cc));
    };
    float sg[4], rp[4], rpr[4], rpa[4], rr[4], pp[4];
    q.load(S, row, sg);
    if (active) {
        q.load(trp, row, rp);
        q.right(trp, row, rp, rpr);
        q.load(trp, above, rpa);
        q.load(trr, row, rr);
        q.load(tpp, row, pp);
    }
    if ((mode & 1) && active) {
        float sl[4], ppl[4], d[4], cc[4];
        q.left(S, row, sg, sl);
        q.left(tpp, row, pp, ppl);
        q.load(dv, row, d);
        if (ph.stabilize == 1) q.load(corr_phi, row, cc);
        const float invrmed = t.InvRmed[i], two = t.TwoOverDRa2[i], r1 = t.RinfSq[i + 1],
                    r0 = t.RinfSq[i];
#pragma unroll
        QUAD {
            const float sa = 0.5f * (sg[k] + sl[k]);
            const float fac = __fdividef(dt * invrmed, sa);
            const float rhs = two * (r1 * rpa[k] - r0 * rp[k]) + (pp[k] - ppl[k]) * g.invdphi;
            // the fused form is spelled out so that every kernel built from
            // this body rounds the update the same way
            if (ph.stabilize == 1)
                d[k] += stabilized(fac * rhs, cc[k]);
            else
                d[k] = fmaf(fac, rhs, d[k]);
        }
        q.store(dv, row, d);
        if (i >= 2) {
            float sb[4], rrb[4], ppb[4], v[4];
            q.load(S, below, sb);
            q.load(trr, below, rrb);
            q.load(tpp, below, ppb);
            q.load(vr, row, v);
            if (ph.stabilize == 1) q.load(corr_r, row, cc);
            const float twos = t.TwoOverRmedSum[i], rm = t.Rmed[i], rmb = t.Rmed[i - 1],
                        invdr = t.InvDiffRmed[i];
#pragma unroll
            QUAD {
                const float sa = 0.5f * (sg[k] + sb[k]);
                const float fac = __fdividef(dt, sa) * ph.rvf * twos;
                const float rhs = (rm * rr[k] - rmb * rrb[k]) * invdr +
                                  (rpr[k] - rp[k]) * g.invdphi - 0.5f * (pp[k] + ppb[k]);
                if (ph.stabilize == 1)
                    v[k] += stabilized(fac * rhs, cc[k]);
                else
                    v[k] = fmaf(fac, rhs, v[k]);
            }
            q.store(vr, row, v);
        }
    }
    if (!(mode & 6) || !ph.adiabatic) return;
    float qp[4] = {}, qm[4] = {}, e[4];
    q.load(E, row, e);
    if (active) {
        if (ph.cooling_beta) {
            float s0[4], e0[4];
            if (ph.beta_ref == 1) {
                q.load(S0, row, s0);
                q.load(E0, row, e0);
            }
            const float emodel = t.EModel[i], omega = t.OmegaK[i];
#pragma unroll
            QUAD {
                float dE = e[k];
                if (ph.beta_ref == 1) dE -= __fdividef(e0[k], s0[k]) * sg[k];
                else if (ph.beta_ref == 2) dE -= emodel * sg[k];
                else if (ph.beta_ref == 3) dE -= sg[k] * ph.emin_fac;
                qm[k] = dE * omega * beta_inv;
            }
        }
        if (ph.heating_viscous) {
            float n[4], dd[4], rpar[4];
            q.load(nu, row, n);
            q.load(divv, row, dd);
            q.right(trp, above, rpa, rpar);
#pragma unroll
            QUAD {
                if (n[k] != 0.f) {
                    const float trpa = 0.25f * (rp[k] + rpa[k] + rpr[k] + rpar[k]);
                    const float a = rr[k], b2 = pp[k];
                    float u = __fdividef(a * a + 2.f * trpa * trpa + b2 * b2, 2.f * n[k] * sg[k]);
                    u += (2.f / 9.f) * n[k] * sg[k] * dd[k] * dd[k];
                    qp[k] = u * ph.hvf;
                }
            }
        }
        float h[4];
        q.load(H, row, h);
#pragma unroll
        QUAD {
            // radiative alpha: 1 + 8 sigma_SB / c * H * x^4 e^3 with
            // x = mu (gamma-1) / (R sigma), evaluated as x * (x e)^3
            const float x = __fdividef(ph.mu_gm1_over_R, sg[k]);
            const float xe = x * e[k];
            const float alpha = 1.f + h[k] * ph.cool_const * x * (xe * xe * xe);
            const float ia = __frcp_rn(alpha);
            qp[k] *= ia;
            qm[k] *= ia;
        }
    }
    if (mode & 4) {
        float en[4];
#pragma unroll
        QUAD {
            en[k] = e[k];
            if (active) {
                en[k] = e[k] + dt * (qp[k] - qm[k]);
                if (sg[k] < ph.sigma_floor10) {
                    qm[k] = qp[k];
                    en[k] = 0.f;
                }
            }
            en[k] = tfloor(en[k], sg[k], ph);
        }
        q.store(E, row, en);
    }
    q.store(qplus, row, qp);
    q.store(qminus, row, qm);
}

// ghost rings (boundary_conditions.cpp:65-114); v_phi hooks work on the
// residual, with the reference-profile offsets per ring
__device__ __forceinline__ void ghost_f(float *x, const float *x0, int kind, int outer, int vec,
                                        int nr, int nz, int j, float kep_value, float zg_offset,
                                        const float *val, const float *nu)
{
    const int irad = vec ? nr : nr - 1;
    const int edge = outer ? irad : 0;
    const int next = outer ? irad - 1 : 1;
    switch (kind) {
    case 1:
        if (!outer) {
            if (vec) {
                x[CELL(0, j)] = x[CELL(2, j)];
                x[CELL(1, j)] = x[CELL(2, j)];
            } else {
                x[CELL(0, j)] = x[CELL(1, j)] + zg_offset;
            }
        } else {
            if (vec) {
                x[CELL(irad, j)] = x[CELL(irad - 2, j)];
                x[CELL(irad - 1, j)] = x[CELL(irad - 2, j)];
            } else {
                x[CELL(irad, j)] = x[CELL(irad - 1, j)] + zg_offset;
            }
        }
        break;
    case 2:
        if (!outer) {
            const float v2 = x[CELL(2, j)];
            x[CELL(1, j)] = v2 > 0.f ? 0.f : v2;
            x[CELL(0, j)] = v2 > 0.f ? 0.f : v2;
        } else {
            const float v2 = x[CELL(irad - 2, j)];
            x[CELL(irad - 1, j)] = v2 < 0.f ? 0.f : v2;
            x[CELL(irad, j)] = v2 < 0.f ? 0.f : v2;
        }
        break;
    case 3:
        x[CELL(edge, j)] = x0[CELL(edge, j)];
        if (vec) x[CELL(next, j)] = x0[CELL(next, j)];
        break;
    case 4:
        x[CELL(edge, j)] = kep_value;
        break;
    case 5:   // disk model
    case 10:  // balanced (residual)
        x[CELL(edge, j)] = val[0];
        break;
    case 6:  // reflecting
        x[CELL(edge, j)] = -x[CELL(outer ? irad - 2 : 2, j)];
        x[CELL(next, j)] = 0.f;
        break;
    case 7: {  // viscous outflow (inner edge)
        const float Nu = 0.5f * (nu[CELL(0, j)] + nu[CELL(1, j)]);
        x[CELL(1, j)] = val[1] * Nu;
        x[CELL(0, j)] = val[0] * Nu;
        break;
    }
    case 8:  // Keplerian radial
        x[CELL(edge, j)] = val[0];
        x[CELL(next, j)] = val[1];
        break;
    case 9:  // zero shear on the residual: ratio * dv_active + offset
        x[CELL(edge, j)] = fmaf(val[0], x[CELL(next, j)], val[1]);
        break;
    default:
        break;
    }
}

// hook part (0 .. 7: field, then edge) of column j; the hooks are independent
// (each writes the ghost rings of its field and edge)
constexpr int kGhostParts = 8;
__device__ __forceinline__ void ghost_col(const GeoF &g, const BcF &bc, const StateF &s, int j,
                                          int part)
{
    const int nz = g.nz, nr = g.nr, outer = part & 1;
    switch (part >> 1) {
    case 0: {
        const int kind = outer ? bc.sigma_out : bc.sigma_in;
        const float *val = outer ? bc.val_out[0] : bc.val_in[0];
        ghost_f(s.sigma, s.sigma0, kind, outer, 0, nr, nz, j, 0.f, 0.f, val, bc.nu);
        // low part of sigma: copied by zero-gradient, cleared by reference hooks,
        // the disk model's own low part
        const int e = outer ? nr - 1 : 0, n = outer ? nr - 2 : 1;
        if (kind == 1) s.sigma_lo[CELL(e, j)] = s.sigma_lo[CELL(n, j)];
        else if (kind == 3) s.sigma_lo[CELL(e, j)] = 0.f;
        else if (kind == 5) s.sigma_lo[CELL(e, j)] = val[1];
        break;
    }
    case 1:
        ghost_f(s.energy, s.energy0, outer ? bc.energy_out : bc.energy_in, outer, 0, nr, nz, j,
                0.f, 0.f, outer ? bc.val_out[1] : bc.val_in[1], bc.nu);
        break;
    case 2:
        ghost_f(s.vr, s.vr0, outer ? bc.vr_out : bc.vr_in, outer, 1, nr, nz, j, 0.f, 0.f,
                outer ? bc.val_out[2] : bc.val_in[2], bc.nu);
        break;
    default:
        ghost_f(s.dv, s.dv0, outer ? bc.vaz_out : bc.vaz_in, outer, 0, nr, nz, j,
                outer ? bc.kep_out : bc.kep_in, outer ? bc.zg_out : bc.zg_in,
                outer ? bc.val_out[3] : bc.val_in[3], bc.nu);
        break;
    }
}

// ---------------------------------------------------------------------------
// radial transport (TransportEuler.cpp:138-167, 349-406, 545-620) with the
// residual angular momentum: quantities 0,1 radial momenta, 2,3 residual
// angular momenta sigma r dv, [4 energy], last sigma.  The angular-momentum
// slopes and the limiter act on the total specific angular momentum
// J_K + r dv (J_K = r v_K per ring), the upwind star value is kept relative to
// J_K of the upwind ring, and the Keplerian part J_K * mass-flux enters the
// residual update through the per-ring differences of J_K.  One thread walks
// column j through rings i0 .. i0 + chunk - 1 with a rolling window.
// ---------------------------------------------------------------------------
template <int NQ>
__device__ __forceinline__ void rad_ring_f(int i, int j, int nz, const float *S, const float *vr,
                                           const float *dv, const float *E, const TablesF &t,
                                           float *w)
{
    const float sg = S[CELL(i, j)];
    const float r = t.Rmed[i];
    w[0] = vr[CELL(i + 1, j)];
    w[1] = vr[CELL(i, j)];
    w[2] = dv[CELL(i, jnext(j, nz))] * r;
    w[3] = dv[CELL(i, j)] * r;
    if (NQ == 5) w[4] = __fdividef(E[CELL(i, j)], sg);
    w[NQ] = sg;
}

// asks L2 for a line; no effect on any value
__device__ __forceinline__ void prefetch_l2(const float *p)
{
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

template <int NQ>
__device__ __forceinline__ void radial_col(const GeoF &g, const TablesF &t, float dt, int mc,
                                           int chunk, const float *__restrict__ S,
                                           const float *__restrict__ vr,
                                           const float *__restrict__ dv,
                                           const float *__restrict__ E, float *__restrict__ m0,
                                           float *__restrict__ m1, float *__restrict__ m2,
                                           float *__restrict__ m3, float *__restrict__ E_out,
                                           float *__restrict__ S_out,
                                           const float *__restrict__ S_lo,
                                           float *__restrict__ S_lo_out, int i0, int j)
{
    constexpr int NW = NQ + 1;
    const int nz = g.nz, nr = g.nr;
    if (i0 >= nr) return;
    const int i1 = min(i0 + chunk, nr);
    const float dtdphi = dt * g.dphi;

    // upward difference of ring k (total slope for the angular momenta)
    auto updiff = [&](int k, const float *wlo, const float *whi, int q) -> float {
        float d = (whi[q] - wlo[q]) * t.InvDiffRmed[k + 1];
        if (q == 2 || q == 3) d += t.JSlope[k];
        return d;
    };
    auto lim = [&](int ring, float up, float down) -> float {
        if (ring <= 0 || ring >= nr - 1) return 0.f;
        return lim_f(up, down, mc);
    };

    float wa[NW] = {}, wb[NW] = {}, wn[NW] = {}, da[NW] = {}, db[NW] = {}, ub[NW] = {};
    {
        float wm2[NW] = {};
        const int r0 = i0 - 1;
        if (r0 - 1 >= 0) rad_ring_f<NQ>(r0 - 1, j, nz, S, vr, dv, E, t, wm2);
        if (r0 >= 0) rad_ring_f<NQ>(r0, j, nz, S, vr, dv, E, t, wa);
        rad_ring_f<NQ>(i0, j, nz, S, vr, dv, E, t, wb);
        const bool has_next = i0 + 1 < nr;
        if (has_next) rad_ring_f<NQ>(i0 + 1, j, nz, S, vr, dv, E, t, wn);
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            const float downa = (r0 - 1 >= 0) ? updiff(r0 - 1, wm2, wa, q) : 0.f;
            const float upa = (r0 >= 0) ? updiff(r0, wa, wb, q) : 0.f;
            da[q] = r0 >= 0 ? lim(r0, upa, downa) : 0.f;
            const float upb = has_next ? updiff(i0, wb, wn, q) : 0.f;
            db[q] = lim(i0, upb, upa);
            ub[q] = upb;
        }
    }
    float flux_prev[NW] = {};
    float kep_prev = 0.f;  // Keplerian term of ring k-1 from interface k-1
    for (int k = i0; k <= i1; ++k) {
        float flux[NW];
        float kep_lower = 0.f, kep_upper = 0.f;
        if (k == 0 || k >= nr) {
#pragma unroll
            for (int q = 0; q < NW; ++q) flux[q] = 0.f;
        } else {
            const float v = vr[CELL(k, j)];
            const float base = dtdphi * t.Rinf[k];
            const float vdt = v * dt;
            float sstar;
            if (v > 0.f) {
                const float f = (t.DRmed[k] - vdt) * 0.5f;
                sstar = wa[NQ] + f * da[NQ];
#pragma unroll
                for (int q = 0; q < NQ; ++q) flux[q] = base * (wa[q] + f * da[q]) * sstar * v;
            } else {
                const float f = (t.DRmed[k + 1] + vdt) * 0.5f;
                sstar = wb[NQ] - f * db[NQ];
#pragma unroll
                for (int q = 0; q < NQ; ++q) flux[q] = base * (wb[q] - f * db[q]) * sstar * v;
            }
            const float fs = base * sstar * v;
            flux[NQ] = fs;
            // J_K(upwind) - J_K(ring) times the mass flux, for the ring above
            // (inflow from below) and the ring below (outflow upwards)
            if (v > 0.f) kep_upper = t.DJ[k] * fs;
            else kep_lower = -t.DJ[k] * fs;
        }
        if (k > i0) {
            // ring k-1's update; its conserved values are formed here from
            // its specific values (wa, the products rounded as stored
            // values) and its energy re-read, so that the walk carries none
            // of them
            const int i = k - 1;
            const float invs = t.InvSurf[i];
            const size_t c = CELL(i, j);
            const float sa = wa[NQ];
            m0[c] = __fmul_rn(sa, wa[0]) + (flux_prev[0] - flux[0]) * invs;
            m1[c] = __fmul_rn(sa, wa[1]) + (flux_prev[1] - flux[1]) * invs;
            m2[c] = __fmul_rn(sa, wa[2]) + (flux_prev[2] + kep_prev - flux[2] - kep_lower) * invs;
            m3[c] = __fmul_rn(sa, wa[3]) + (flux_prev[3] + kep_prev - flux[3] - kep_lower) * invs;
            if (NQ == 5) E_out[c] = E[c] + (flux_prev[4] - flux[4]) * invs;
            float hi = sa, lo = S_lo[c];
            comp_add(hi, lo, (flux_prev[NQ] - flux[NQ]) * invs);
            S_out[c] = hi;
            S_lo_out[c] = lo;
        }
        if (k < i1) {
#pragma unroll
            for (int q = 0; q < NW; ++q) flux_prev[q] = flux[q];
            kep_prev = kep_upper;
            // the ring after the next comes from DRAM, whose latency the walk
            // waited for (2048 x 6144: 0.302 -> 0.277 ms; one ring further on
            // 0.278, three 0.285; a batch of 16 disks 0.174 -> 0.157)
            if (k + 3 <= i1 && k + 3 < nr) {
                const size_t c = CELL(k + 3, j);
                prefetch_l2(S + c);
                prefetch_l2(dv + c);
                prefetch_l2(vr + c + nz);
                if (NQ == 5) prefetch_l2(E + c);
                prefetch_l2(S_lo + c);
            }
            const bool more = k + 2 < nr;
            float w2[NW] = {};
            if (more) rad_ring_f<NQ>(k + 2, j, nz, S, vr, dv, E, t, w2);
#pragma unroll
            for (int q = 0; q < NW; ++q) {
                wa[q] = wb[q];
                da[q] = db[q];
                wb[q] = wn[q];
                const float up = more ? updiff(k + 1, wn, w2, q) : 0.f;
                db[q] = lim(k + 1, up, ub[q]);
                ub[q] = up;
                wn[q] = w2[q];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// azimuthal transport with FARGO (TransportEuler.cpp:174-304, 416-466,
// 630-664): FP32 advection, FP64 ring mean and shift phase.  The residual
// angular momentum is advected like any specific quantity (J_K is constant on
// a ring, so its part cancels exactly).  One block per ring; thread tid owns
// cells tid + n * blockDim.x, n < PER, which must cover the ring.  Each
// quantity takes three barriers: specific values, slopes, fluxes (a separate
// flux array lets the update read them while the next quantity starts).
// ---------------------------------------------------------------------------
template <int PER, int NQ>
__device__ __forceinline__ void ring_pass_f(float *S, float *W, float *D, float *F, float *X,
                                            float *const *qrow, const float *v, float *slo,
                                            float dt, float dxtheta, float half_invdx,
                                            float dxrad_invsurf, int nz, int mc)
{
    const int tid = threadIdx.x, bs = blockDim.x;
    // per face: 1 / sigma of the cell and dxrad S* v / Surf, the factor every
    // quantity's flux shares; kept in the X array up to 4 cells per thread
    // (short rings, shared memory to spare) and in registers beyond
    constexpr bool XS = PER <= 4;
    float invs[PER], cfr[XS ? 1 : PER];
    auto cf = [&](int n, int j) -> float & { return XS ? X[j] : cfr[n]; };
#pragma unroll
    for (int n = 0; n < PER; ++n) {
        const int j = tid + n * bs;
        if (j < nz) {
            const int jp = j == nz - 1 ? 0 : j + 1, jm = j == 0 ? nz - 1 : j - 1;
            D[j] = __fmul_rn(lim_f(__fsub_rn(S[jp], S[j]), __fsub_rn(S[j], S[jm]), mc), half_invdx);
            invs[n] = __frcp_rn(S[j]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < PER; ++n) {
        const int j = tid + n * bs;
        if (j < nz) {
            const int jm = j == 0 ? nz - 1 : j - 1;
            const float vv = v[n];
            const float ksi = __fmul_rn(vv, dt);
            const float ss = ksi > 0.f ? star_pos(S[jm], D[jm], dxtheta, ksi)
                                       : star_neg(S[j], D[j], dxtheta, ksi);
            cf(n, j) = __fmul_rn(__fmul_rn(dxrad_invsurf, ss), vv);
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        float *Q = qrow[q];
#pragma unroll
        for (int n = 0; n < PER; ++n) {
            const int j = tid + n * bs;
            if (j < nz) W[j] = __fmul_rn(Q[j], invs[n]);
        }
        __syncthreads();
#pragma unroll
        for (int n = 0; n < PER; ++n) {
            const int j = tid + n * bs;
            if (j < nz) {
                const int jp = j == nz - 1 ? 0 : j + 1, jm = j == 0 ? nz - 1 : j - 1;
                D[j] = __fmul_rn(lim_f(__fsub_rn(W[jp], W[j]), __fsub_rn(W[j], W[jm]), mc), half_invdx);
            }
        }
        __syncthreads();
#pragma unroll
        for (int n = 0; n < PER; ++n) {
            const int j = tid + n * bs;
            if (j < nz) {
                const int jm = j == 0 ? nz - 1 : j - 1;
                const float ksi = __fmul_rn(v[n], dt);
                const float qs = ksi > 0.f ? star_pos(W[jm], D[jm], dxtheta, ksi)
                                           : star_neg(W[j], D[j], dxtheta, ksi);
                F[j] = __fmul_rn(qs, cf(n, j));
            }
        }
        __syncthreads();
#pragma unroll
        for (int n = 0; n < PER; ++n) {
            const int j = tid + n * bs;
            if (j < nz) Q[j] = __fadd_rn(Q[j], __fsub_rn(F[j], F[j == nz - 1 ? 0 : j + 1]));
        }
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < PER; ++n) {
        const int j = tid + n * bs;
        if (j < nz) F[j] = cf(n, j);
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < PER; ++n) {
        const int j = tid + n * bs;
        if (j < nz) {
            float sn = S[j];
            comp_add(sn, slo[n], F[j] - F[j == nz - 1 ? 0 : j + 1]);
            S[j] = sn;
        }
    }
    __syncthreads();
}

// The uniform pass of FARGO (QuantitiesAdvection with the ring's residual
// shift velocity, TransportEuler.cpp:292-304) in difference form.  The whole
// ring has one upwind direction, so with u the upwind cell of face j
// (j - 1 for a positive shift, j otherwise) and a the interpolation distance
// (dx - ksi, or -(dx + ksi)), face j's star value is X_u + a D_u and cell j
// changes by dxrad v invsurf (q*_j S*_j - q*_{j+1} S*_{j+1})
//   = dxrad v invsurf (q*_j dS*_j + S*_{j+1} dq*_j),
//   dS*_j = (S_u - S_{u+1}) + a (D_u - D_{u+1}),  dq*_j likewise.
// This is the flux form's arithmetic regrouped: forming the neighbour
// differences first keeps FP32's rounding at the size of the changes, where
// the flux form rounds at the size of the fluxes, up to half of the ring's
// content per step, and repeats the same rounding pattern every step.
// dS* goes to the X array (up to 4 cells per thread) or registers, S*_{j+1}
// to the F array; c is dxrad v invsurf and a the interpolation distance.
template <int PER, int NQ>
__device__ __forceinline__ void ring_pass_uniform_f(float *S, float *W, float *D, float *F,
                                                    float *X, float *const *qrow, float *slo,
                                                    bool pos, float a, float c, float half_invdx,
                                                    int nz, int mc)
{
    const int tid = threadIdx.x, bs = blockDim.x;
    constexpr bool XS = PER <= 4;
    float invs[PER], dssr[XS ? 1 : PER];
    auto dss = [&](int n, int j) -> float & { return XS ? X[j] : dssr[n]; };
#pragma unroll
    for (int n = 0; n < PER; ++n) {
        const int j = tid + n * bs;
        if (j < nz) {
            const int jp = j == nz - 1 ? 0 : j + 1, jm = j == 0 ? nz - 1 : j - 1;
            D[j] = __fmul_rn(lim_f(__fsub_rn(S[jp], S[j]), __fsub_rn(S[j], S[jm]), mc), half_invdx);
            invs[n] = __frcp_rn(S[j]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < PER; ++n) {
        const int j = tid + n * bs;
        if (j < nz) {
            const int jp = j == nz - 1 ? 0 : j + 1, jm = j == 0 ? nz - 1 : j - 1;
            const int u = pos ? jm : j, u1 = pos ? j : jp;
            dss(n, j) = star_diff(S[u], S[u1], D[u], D[u1], a);
            F[j] = star_at(S[u1], D[u1], a);
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        float *Q = qrow[q];
#pragma unroll
        for (int n = 0; n < PER; ++n) {
            const int j = tid + n * bs;
            if (j < nz) W[j] = __fmul_rn(Q[j], invs[n]);
        }
        __syncthreads();
#pragma unroll
        for (int n = 0; n < PER; ++n) {
            const int j = tid + n * bs;
            if (j < nz) {
                const int jp = j == nz - 1 ? 0 : j + 1, jm = j == 0 ? nz - 1 : j - 1;
                D[j] = __fmul_rn(lim_f(__fsub_rn(W[jp], W[j]), __fsub_rn(W[j], W[jm]), mc), half_invdx);
            }
        }
        __syncthreads();
#pragma unroll
        for (int n = 0; n < PER; ++n) {
            const int j = tid + n * bs;
            if (j < nz) {
                const int jp = j == nz - 1 ? 0 : j + 1, jm = j == 0 ? nz - 1 : j - 1;
                const int u = pos ? jm : j, u1 = pos ? j : jp;
                const float qs = star_at(W[u], D[u], a);
                const float dqs = star_diff(W[u], W[u1], D[u], D[u1], a);
                Q[j] = uniform_update(Q[j], c, qs, dss(n, j), F[j], dqs);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int n = 0; n < PER; ++n) {
        const int j = tid + n * bs;
        if (j < nz) {
            float sn = S[j];
            comp_add(sn, slo[n], __fmul_rn(c, dss(n, j)));
            S[j] = sn;
        }
    }
    __syncthreads();
}

// Shared memory of azimuthal_ring: ring-long work arrays for sigma, the
// specific quantity, its slope and the flux, a fifth for the per-face factors
// on rings up to 2048 cells (where at most 4 cells per thread leave no
// registers for them), plus the nq quantity rows when STAGE (then every row
// is read from HBM once, up front, the passes work in shared memory and the
// rows go back once at the end).
__host__ __device__ constexpr int azimuthal_work_rows(int nz) { return nz <= 2048 ? 5 : 4; }
__host__ __device__ constexpr size_t azimuthal_smem_floats(int nz, int nq, bool stage)
{
    return (size_t)(azimuthal_work_rows(nz) + (stage ? nq : 0)) * (size_t)nz;
}

// smf: azimuthal_smem_floats(nz, nq, STAGE) floats of shared memory; redf: 33
// floats, redl: 33 long longs (shared memory)
template <int PER, int NQ, bool STAGE>
__device__ __forceinline__ void azimuthal_ring(const GeoF &g, const TablesF &t, double dt, int mc,
                                               int fast, const float *__restrict__ dv,
                                               float *m0, float *m1, float *m2, float *m3,
                                               float *E, float *S, float *S_lo, int i, float *smf,
                                               float *redf, long long *redl, int *ring_shift)
{
    const int nz = g.nz;
    const int tid = threadIdx.x, bs = blockDim.x;
    const size_t row = (size_t)i * nz;
    float *Sr = smf, *W = smf + nz, *D = smf + 2 * nz, *Fx = smf + 3 * nz;
    // the per-face array exists when PER <= 4, which needs nz <= 4 x 512
    float *X = smf + 4 * nz;
    const int wr = azimuthal_work_rows(nz);
    float *grow[5] = {m0 + row, m1 + row, m2 + row, m3 + row, E + row};
    float *qrow[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) qrow[q] = STAGE ? smf + (size_t)(wr + q) * nz : grow[q];

    float vown[PER], slo[PER];
    float amax = 0.f;
#pragma unroll
    for (int n = 0; n < PER; ++n) {
        const int j = tid + n * bs;
        if (j < nz) {
            vown[n] = dv[row + j];
            amax = fmaxf(amax, fabsf(vown[n]));
            Sr[j] = S[row + j];
            slo[n] = S_lo[row + j];
            if (STAGE) {
#pragma unroll
                for (int q = 0; q < NQ; ++q) qrow[q][j] = grow[q][j];
            }
        }
    }
    // ring mean of v_phi, independent of the block's shape, and the FARGO
    // shift phase in FP64 (:174-236)
    const int ks = exact_sum_scale(amax, nz, redf);
    long long part = 0;
#pragma unroll
    for (int n = 0; n < PER; ++n)
        if (tid + n * bs < nz) part += to_fixed(vown[n], ks);
    const double mean_dv = exact_sum_result(part, ks, redl) / (double)nz;
    // the ring's mean frame velocity (the residual is about the inertial
    // Keplerian speed)
    const double vmean = (t.Vref_d[i] - t.Rmed_d[i] * g.omega_frame) + mean_dv;
    const double Ntilde = vmean * t.InvRmed_d[i] * dt * g.invdphi_d;
    const double Nround = floor(Ntilde + 0.5);
    const int nshift = (int)Nround;
    const float vt = (float)((Ntilde - Nround) * t.Rmed_d[i] * (1.0 / dt) * g.dphi_d);
    const float mdv = (float)mean_dv;
#pragma unroll
    for (int n = 0; n < PER; ++n) {
        const int j = tid + n * bs;
        if (j < nz) {
            // residual about the ring mean (compute_residual_velocity, :194-205)
            float vres = vown[n] - mdv;
            if (!fast) vres = vt + vres;
            vown[n] = vres;
        }
    }
    const float dxtheta = g.dphi * t.Rmed[i];
    const float half_invdx = 0.5f / dxtheta;
    const float dxrad = t.DRsup[i] * (float)dt;
    const float invsurf = t.InvSurf[i];
    ring_pass_f<PER, NQ>(Sr, W, D, Fx, X, qrow, vown, slo, (float)dt, dxtheta, half_invdx,
                         dxrad * invsurf, nz, mc);
    if (fast) {
        const float ksi = vt * (float)dt;
        const bool pos = ksi > 0.f;
        ring_pass_uniform_f<PER, NQ>(Sr, W, D, Fx, X, qrow, slo, pos,
                                     pos ? dxtheta - ksi : -(dxtheta + ksi),
                                     dxrad * vt * invsurf, half_invdx, nz, mc);
    }
    // AdvectSHIFT (:238-268) is the velocity rebuild's: it reads cell j of
    // this ring from cell j - nshift, so the rows go back unshifted (the
    // quantities are already in place unless staged)
#pragma unroll
    for (int n = 0; n < PER; ++n) {
        const int j = tid + n * bs;
        if (j < nz) {
            S[row + j] = Sr[j];
            S_lo[row + j] = slo[n];
        }
    }
    if (STAGE) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
#pragma unroll
            for (int n = 0; n < PER; ++n) {
                const int j = tid + n * bs;
                if (j < nz) grow[q][j] = qrow[q][j];
            }
        }
    }
    if (tid == 0) ring_shift[i] = ((nshift % nz) + nz) % nz;
    // the caller may reuse smf for the next ring
    __syncthreads();
}

// ---------------------------------------------------------------------------
// The same ring transport with the ring in registers: thread tid owns the
// contiguous cells j0 = tid PER .. j0 + PER - 1 (nz = PER blockDim.x, PER a
// multiple of 4), loads and stores them as 128-bit words, and computes every
// stencil from registers.  The only cross-thread step per transported
// quantity is one exchange of segment ends: each thread publishes its first
// two and last two values, and after one barrier reads the two cells left of
// its segment and the two right of it; with them it forms the slopes of
// cells j0 - 1 .. j0 + PER and the fluxes of faces j0 .. j0 + PER itself, so
// no slope or flux crosses threads.  The exchange area is double-buffered:
// a thread writing buffer b for the next exchange has passed the barrier of
// the exchange in between, which every thread reaches only after reading
// buffer b, so no write overtakes a read.  Every cell's arithmetic is the
// strided kernel's (ring_pass_f, ring_pass_uniform_f, the exact-sum ring mean,
// the shift phase), expression for expression, so both give the same bits.
//
// Shared memory (rb_smem_floats): the NQ transported rows between the two
// passes (staged coalesced from HBM; the last pass writes each segment back
// to its row in place, the integer shift being the velocity rebuild's) and
// 2 x 5 x blockDim.x floats for the exchanges.
// ---------------------------------------------------------------------------
// threads per ring block of the register-blocked kernel: 16 cells per thread
// need more registers than 128 (the budget at 512 threads)
__host__ __device__ constexpr int rb_max_threads(int per) { return per >= 16 ? 384 : 512; }
__host__ __device__ constexpr size_t rb_smem_floats(int nz, int nq, int threads)
{
    return (size_t)nq * (size_t)nz + (size_t)10 * (size_t)threads;
}
// whether a ring of nz cells splits into segments of per cells within the kernel's
// bound of threads and max_smem bytes
__host__ __device__ inline bool rb_fits(int nz, int nq, int per, size_t max_smem)
{
    if (nz % per != 0) return false;
    const int th = nz / per;
    return th <= rb_max_threads(per) &&
           rb_smem_floats(nz, nq, th) * sizeof(float) <= max_smem;
}
template <int PER, int NQ>
__device__ __forceinline__ void azimuthal_ring_rb(const GeoF &g, const TablesF &t, double dt,
                                                  int mc, int fast, const float *__restrict__ dv,
                                                  float *m0, float *m1, float *m2, float *m3,
                                                  float *E, float *S, float *S_lo, int i,
                                                  float *smf, float *redf, long long *redl,
                                                  int *ring_shift)
{
    static_assert(PER % 4 == 0 && PER >= 4, "segments of whole 128-bit words");
    const int nz = g.nz;  // == PER * blockDim.x
    const int tid = threadIdx.x, bs = blockDim.x;
    const size_t row = (size_t)i * nz;
    const int j0 = tid * PER;
    const int left = tid == 0 ? bs - 1 : tid - 1, right = tid == bs - 1 ? 0 : tid + 1;
    float *qsm = smf;                               // NQ rows
    float *xs = smf + (size_t)NQ * nz;              // [2][5][bs]
    float *grow[5] = {m0 + row, m1 + row, m2 + row, m3 + row, E + row};
    int buf = 0;
    // publishes a0, a1 (first two), a2, a3 (last two) and a4; returns the
    // left neighbour's last two (l2, l3), the right neighbour's first two
    // (r0, r1) and its a4 (r4)
    auto exchange = [&](float a0, float a1, float a2, float a3, float a4, float &l2, float &l3,
                        float &r0, float &r1, float &r4) {
        float *x = xs + (size_t)buf * 5 * bs;
        x[tid] = a0;
        x[bs + tid] = a1;
        x[2 * bs + tid] = a2;
        x[3 * bs + tid] = a3;
        x[4 * bs + tid] = a4;
        __syncthreads();
        l2 = x[2 * bs + left];
        l3 = x[3 * bs + left];
        r0 = x[right];
        r1 = x[bs + right];
        r4 = x[4 * bs + right];
        buf ^= 1;
    };
    auto load_seg = [&](const float *src, float *dst) {
#pragma unroll
        for (int k = 0; k < PER / 4; ++k) {
            const float4 w = reinterpret_cast<const float4 *>(src + j0)[k];
            dst[4 * k] = w.x;
            dst[4 * k + 1] = w.y;
            dst[4 * k + 2] = w.z;
            dst[4 * k + 3] = w.w;
        }
    };
    auto store_seg = [&](float *dst, const float *src) {
#pragma unroll
        for (int k = 0; k < PER / 4; ++k)
            reinterpret_cast<float4 *>(dst + j0)[k] =
                make_float4(src[4 * k], src[4 * k + 1], src[4 * k + 2], src[4 * k + 3]);
    };

    // the transported rows into shared memory (coalesced), the own segment of
    // v_phi and of the sigma pair into registers
#pragma unroll
    for (int q = 0; q < NQ; ++q)
        for (int j = tid; j < nz; j += bs) qsm[(size_t)q * nz + j] = grow[q][j];
    float v[PER + 1], s[PER], slo[PER];
    load_seg(dv + row, v);
    load_seg(S + row, s);
    load_seg(S_lo + row, slo);
    float amax = 0.f;
#pragma unroll
    for (int n = 0; n < PER; ++n) amax = fmaxf(amax, fabsf(v[n]));
    // ring mean of v_phi (exact integer sum: the same bits for any ownership)
    // and the FARGO shift phase in FP64 (:174-236)
    const int ks = exact_sum_scale(amax, nz, redf);
    long long part = 0;
#pragma unroll
    for (int n = 0; n < PER; ++n) part += to_fixed(v[n], ks);
    const double mean_dv = exact_sum_result(part, ks, redl) / (double)nz;
    const double vmean = (t.Vref_d[i] - t.Rmed_d[i] * g.omega_frame) + mean_dv;
    const double Ntilde = vmean * t.InvRmed_d[i] * dt * g.invdphi_d;
    const double Nround = floor(Ntilde + 0.5);
    const int nshift = (int)Nround;
    const float vt = (float)((Ntilde - Nround) * t.Rmed_d[i] * (1.0 / dt) * g.dphi_d);
    const float mdv = (float)mean_dv;
#pragma unroll
    for (int n = 0; n < PER; ++n) {
        float vres = v[n] - mdv;
        if (!fast) vres = vt + vres;
        v[n] = vres;
    }
    const float dxtheta = g.dphi * t.Rmed[i];
    const float half_invdx = 0.5f / dxtheta;
    const float dxrad = t.DRsup[i] * (float)dt;
    const float invsurf = t.InvSurf[i];
    const float fdt = (float)dt;
    const float dxrad_invsurf = dxrad * invsurf;
    __syncthreads();  // the staged rows are complete

    // values of cells j0 - 2 .. j0 + PER + 1 at index c + 2; slopes of cells
    // j0 - 1 .. j0 + PER at index c + 1
    float X[PER + 4], D[PER + 2], invs[PER];
    auto slopes = [&]() {
#pragma unroll
        for (int c = -1; c <= PER; ++c)
            D[c + 1] = __fmul_rn(lim_f(__fsub_rn(X[c + 3], X[c + 2]), __fsub_rn(X[c + 2], X[c + 1]), mc),
                                 half_invdx);
    };
    auto sigma_ends = [&](float a4, float &r4) {
        float l2, l3, r0, r1;
        exchange(s[0], s[1], s[PER - 2], s[PER - 1], a4, l2, l3, r0, r1, r4);
        X[0] = l2;
        X[1] = l3;
#pragma unroll
        for (int n = 0; n < PER; ++n) X[n + 2] = s[n];
        X[PER + 2] = r0;
        X[PER + 3] = r1;
    };
    auto specific = [&](const float *q) {
#pragma unroll
        for (int n = 0; n < PER; ++n) X[n + 2] = __fmul_rn(q[n], invs[n]);
        float l2, l3, r0, r1, r4;
        exchange(X[2], X[3], X[PER], X[PER + 1], 0.f, l2, l3, r0, r1, r4);
        X[0] = l2;
        X[1] = l3;
        X[PER + 2] = r0;
        X[PER + 3] = r1;
    };

    // QuantitiesAdvection with the residual velocity (ring_pass_f)
    {
        float cf[PER + 1];
        sigma_ends(v[0], v[PER]);  // face j0 + PER takes the right neighbour's velocity
        slopes();
#pragma unroll
        for (int n = 0; n < PER; ++n) invs[n] = __frcp_rn(s[n]);
#pragma unroll
        for (int f = 0; f <= PER; ++f) {
            const float vv = v[f];
            const float ksi = __fmul_rn(vv, fdt);
            const float ss = ksi > 0.f ? star_pos(X[f + 1], D[f], dxtheta, ksi)
                                       : star_neg(X[f + 2], D[f + 1], dxtheta, ksi);
            cf[f] = __fmul_rn(__fmul_rn(dxrad_invsurf, ss), vv);
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            float qv[PER];
            load_seg(qsm + (size_t)q * nz, qv);
            specific(qv);
            slopes();
            float F[PER + 1];
#pragma unroll
            for (int f = 0; f <= PER; ++f) {
                const float ksi = __fmul_rn(v[f], fdt);
                const float qs = ksi > 0.f ? star_pos(X[f + 1], D[f], dxtheta, ksi)
                                           : star_neg(X[f + 2], D[f + 1], dxtheta, ksi);
                F[f] = __fmul_rn(qs, cf[f]);
            }
#pragma unroll
            for (int n = 0; n < PER; ++n) qv[n] = __fadd_rn(qv[n], __fsub_rn(F[n], F[n + 1]));
            // the last pass writes the segment back to its row in place
            store_seg(fast ? qsm + (size_t)q * nz : grow[q], qv);
        }
#pragma unroll
        for (int n = 0; n < PER; ++n) comp_add(s[n], slo[n], cf[n] - cf[n + 1]);
    }
    // the uniform pass in difference form (ring_pass_uniform_f)
    if (fast) {
        const float ksi = vt * fdt;
        const bool pos = ksi > 0.f;
        const float a = pos ? dxtheta - ksi : -(dxtheta + ksi);
        const float c = dxrad * vt * invsurf;
        float dss[PER], Fs[PER];
        float unused;
        sigma_ends(0.f, unused);
        slopes();
#pragma unroll
        for (int n = 0; n < PER; ++n) {
            invs[n] = __frcp_rn(s[n]);
            // cells u (upwind of face j) and u1 (of face j + 1): n - 1 and n
            // for a positive shift, n and n + 1 otherwise (X index + 2, D
            // index + 1); both candidates are read and one is selected, so
            // the arrays stay in registers
            const float xu = pos ? X[n + 1] : X[n + 2], xu1 = pos ? X[n + 2] : X[n + 3];
            const float du = pos ? D[n] : D[n + 1], du1 = pos ? D[n + 1] : D[n + 2];
            dss[n] = star_diff(xu, xu1, du, du1, a);
            Fs[n] = star_at(xu1, du1, a);
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            float qv[PER];
            load_seg(qsm + (size_t)q * nz, qv);
            specific(qv);
            slopes();
#pragma unroll
            for (int n = 0; n < PER; ++n) {
                const float xu = pos ? X[n + 1] : X[n + 2], xu1 = pos ? X[n + 2] : X[n + 3];
                const float du = pos ? D[n] : D[n + 1], du1 = pos ? D[n + 1] : D[n + 2];
                const float qs = star_at(xu, du, a);
                const float dqs = star_diff(xu, xu1, du, du1, a);
                qv[n] = uniform_update(qv[n], c, qs, dss[n], Fs[n], dqs);
            }
            store_seg(grow[q], qv);
        }
#pragma unroll
        for (int n = 0; n < PER; ++n) comp_add(s[n], slo[n], __fmul_rn(c, dss[n]));
    }

    // AdvectSHIFT (:238-268) is the velocity rebuild's: it reads cell j of
    // this ring from cell j - nshift; the last pass wrote the quantities'
    // segments in place, sigma and its low part follow
    store_seg(S + row, s);
    store_seg(S_lo + row, slo);
    if (tid == 0) ring_shift[i] = ((nshift % nz) + nz) % nz;
    // the caller may reuse smf for the next ring
    __syncthreads();
}

// ---------------------------------------------------------------------------
// The same ring transport without barriers: a warp owns a window of 128
// consecutive cells of a ring, four per lane in registers, and writes the 120
// inner ones; the four cells at either end, which both passes of the inner
// cells need, are computed along with them, so that no warp waits for
// another and a ring needs no shared memory.  Neighbours beyond a lane's
// four cells come by shuffles.  The ring means and the shift phase are the
// radial launch's (ring_phase_f), and the output goes to other buffers than the
// input, since neighbouring windows overlap.  Every cell's arithmetic is the
// ring kernels' above, expression for expression: the same bits.
//
// The ring kernels are bound by latency (two or three block barriers per
// quantity and pass, a block of at most 512 threads per SM: issue 29% of the
// cycles, DRAM 10%); this one keeps 24 warps per SM resident and has no
// barrier.  Measured, ms per azimuthal pass (register-blocked or strided
// ring kernel -> this): 2048 x 6144 0.547 -> 0.236, 512 x 1536 0.049 -> 0.021,
// 128 x 384 0.014 -> 0.010, the 64-disk sweep's step 3.84 -> 3.15.  Issue is
// 71% busy, DRAM 29%.
// ---------------------------------------------------------------------------
constexpr int kWinCells = 4;                            // cells per lane
constexpr int kWinInner = 30 * kWinCells;               // cells a warp writes
__host__ __device__ constexpr int windows_of(int nz) { return (nz + kWinInner - 1) / kWinInner; }

// A ring's mean residual velocity and uniform velocity (ComputeConstantResidual,
// TransportEuler.cpp:174-236), and its integer shift, by one warp (the exact
// integer sum of exact_sum_scale / exact_sum_result: the ring kernels' bits).
__device__ __forceinline__ void ring_phase_f(const GeoF &g, const TablesF &t, double dt,
                                             const float *__restrict__ dv, int i, float2 *phase,
                                             int *ring_shift)
{
    const int nz = g.nz, lane = threadIdx.x & 31;
    const float *v = dv + (size_t)i * nz;
    float m = 0.f;
#pragma unroll 8
    for (int j = lane; j < nz; j += 32) m = fmaxf(m, fabsf(v[j]));
    m = __shfl_sync(0xffffffffu, warp_max_f(m), 0);
    int e = 0;
    frexpf(m, &e);
    const int ks = 62 - e - (32 - __clz(nz));
    long long part = 0;
#pragma unroll 8
    for (int j = lane; j < nz; j += 32) part += to_fixed(v[j], ks);
    part = warp_sum_ll(part);
    if (lane == 0) {
        const double mean_dv = ldexp((double)part, -ks) / (double)nz;
        const double vmean = (t.Vref_d[i] - t.Rmed_d[i] * g.omega_frame) + mean_dv;
        const double Ntilde = vmean * t.InvRmed_d[i] * dt * g.invdphi_d;
        const double Nround = floor(Ntilde + 0.5);
        const int nshift = (int)Nround;
        const float vt = (float)((Ntilde - Nround) * t.Rmed_d[i] * (1.0 / dt) * g.dphi_d);
        phase[i] = make_float2((float)mean_dv, vt);
        ring_shift[i] = ((nshift % nz) + nz) % nz;
    }
}

// the rows a window reads and writes (m: momenta, e: energy, s, slo: sigma)
struct WindowRows {
    const float *dv, *m0, *m1, *m2, *m3, *e, *s, *slo;
    float *om0, *om1, *om2, *om3, *oe, *os, *oslo;
    __device__ __forceinline__ const float *in(int q) const
    {
        return q == 0 ? m0 : q == 1 ? m1 : q == 2 ? m2 : q == 3 ? m3 : e;
    }
    __device__ __forceinline__ float *out(int q) const
    {
        return q == 0 ? om0 : q == 1 ? om1 : q == 2 ? om2 : q == 3 ? om3 : oe;
    }
};

template <int NQ>
__device__ __forceinline__ void azimuthal_window(const GeoF &g, const TablesF &t, double dt,
                                                 int mc, int fast, const WindowRows &rows,
                                                 float2 phase, int i, int window)
{
    constexpr unsigned all = 0xffffffffu;
    constexpr int N = kWinCells;
    const int nz = g.nz, lane = threadIdx.x & 31;
    const size_t row = (size_t)i * nz;
    const int base = window * kWinInner + (lane - 1) * N;
    const int valid = lane == 0 || lane == 31 ? 0 : min(N, nz - base);
    const bool aligned = (nz & 3) == 0;  // a lane's cells are one 128-bit word
    int j[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        int b = base + k;
        if (b < 0) b += nz;
        if (b >= nz) b = b - nz < nz ? b - nz : b % nz;
        j[k] = b;
    }
    auto load = [&](const float *p, float *x) {
        if (aligned) {
            const float4 w = *reinterpret_cast<const float4 *>(p + row + j[0]);
            x[0] = w.x; x[1] = w.y; x[2] = w.z; x[3] = w.w;
        } else {
#pragma unroll
            for (int k = 0; k < N; ++k) x[k] = p[row + j[k]];
        }
    };
    auto store = [&](float *p, const float *x) {
        if (aligned) {
            if (valid > 0)
                *reinterpret_cast<float4 *>(p + row + base) = make_float4(x[0], x[1], x[2], x[3]);
        } else {
#pragma unroll
            for (int k = 0; k < N; ++k)
                if (k < valid) p[row + base + k] = x[k];
        }
    };
    auto left = [&](float x) { return __shfl_up_sync(all, x, 1); };
    auto right = [&](float x) { return __shfl_down_sync(all, x, 1); };

    float v[N], s[N], slo[N], next[N];
    load(rows.dv, v);
    load(rows.s, s);
    load(rows.slo, slo);
    load(rows.m0, next);
    // the other rows come from DRAM: ask L2 for them now
#pragma unroll
    for (int q = 1; q < NQ; ++q)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(rows.in(q) + row + j[0]));
    const float mdv = phase.x, vt = phase.y;
#pragma unroll
    for (int n = 0; n < N; ++n) {
        float vres = v[n] - mdv;
        if (!fast) vres = vt + vres;
        v[n] = vres;
    }
    const float dxtheta = g.dphi * t.Rmed[i];
    const float half_invdx = 0.5f / dxtheta;
    const float dxrad = t.DRsup[i] * (float)dt;
    const float invsurf = t.InvSurf[i];
    const float fdt = (float)dt;
    const float dxrad_invsurf = dxrad * invsurf;

    // cells -1 .. 3 of X and of its slopes at index + 1
    auto slopes = [&](float *X, float *D) {
        X[0] = left(X[N]);
        float d[N + 1];
#pragma unroll
        for (int k = 0; k < N; ++k) d[k] = __fsub_rn(X[k + 1], X[k]);
        d[N] = right(d[0]);
#pragma unroll
        for (int k = 0; k < N; ++k) D[k + 1] = __fmul_rn(lim_f(d[k + 1], d[k], mc), half_invdx);
        D[0] = left(D[N]);
    };
    float cf[N + 1], invs[N];
    // the uniform pass: face factors in difference form (ring_pass_uniform_f)
    const float ksi_u = vt * fdt;
    const bool pos = ksi_u > 0.f;
    const float a = pos ? dxtheta - ksi_u : -(dxtheta + ksi_u);
    const float c = dxrad * vt * invsurf;
    float dss[N], Fs[N], invs2[N];
    // X_u, X_u1, D_u, D_u1 of face n, upwind cell u and its right neighbour u1
    auto uniform_sides = [&](float *X, float *D) {
        if (pos) return;
        // cells 0 .. 4 instead of -1 .. 3
        const float xr = right(X[1]), dr = right(D[1]);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            X[k] = X[k + 1];
            D[k] = D[k + 1];
        }
        X[N] = xr;
        D[N] = dr;
    };
    {
        float X[N + 1], D[N + 1];
#pragma unroll
        for (int n = 0; n < N; ++n) X[n + 1] = s[n];
        slopes(X, D);
#pragma unroll
        for (int n = 0; n < N; ++n) {
            invs[n] = __frcp_rn(s[n]);
            const float vv = v[n];
            const float ksi = __fmul_rn(vv, fdt);
            const float ss = ksi > 0.f ? star_pos(X[n], D[n], dxtheta, ksi)
                                       : star_neg(X[n + 1], D[n + 1], dxtheta, ksi);
            cf[n] = __fmul_rn(__fmul_rn(dxrad_invsurf, ss), vv);
        }
        cf[N] = right(cf[0]);
#pragma unroll
        for (int n = 0; n < N; ++n) comp_add(s[n], slo[n], cf[n] - cf[n + 1]);
    }
    if (fast) {
        float X[N + 1], D[N + 1];
#pragma unroll
        for (int n = 0; n < N; ++n) X[n + 1] = s[n];
        slopes(X, D);
        uniform_sides(X, D);
#pragma unroll
        for (int n = 0; n < N; ++n) {
            invs2[n] = __frcp_rn(s[n]);
            dss[n] = star_diff(X[n], X[n + 1], D[n], D[n + 1], a);
            Fs[n] = star_at(X[n + 1], D[n + 1], a);
        }
#pragma unroll
        for (int n = 0; n < N; ++n) comp_add(s[n], slo[n], __fmul_rn(c, dss[n]));
    }
    store(rows.os, s);
    store(rows.oslo, slo);
#pragma unroll 1
    for (int q = 0; q < NQ; ++q) {
        float qv[N], X[N + 1], D[N + 1];
#pragma unroll
        for (int n = 0; n < N; ++n) {
            qv[n] = next[n];
            X[n + 1] = __fmul_rn(qv[n], invs[n]);
        }
        if (q + 1 < NQ) load(rows.in(q + 1), next);
        slopes(X, D);
        float F[N + 1];
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const float ksi = __fmul_rn(v[n], fdt);
            const float qs = ksi > 0.f ? star_pos(X[n], D[n], dxtheta, ksi)
                                       : star_neg(X[n + 1], D[n + 1], dxtheta, ksi);
            F[n] = __fmul_rn(qs, cf[n]);
        }
        F[N] = right(F[0]);
#pragma unroll
        for (int n = 0; n < N; ++n) qv[n] = __fadd_rn(qv[n], __fsub_rn(F[n], F[n + 1]));
        if (fast) {
#pragma unroll
            for (int n = 0; n < N; ++n) X[n + 1] = __fmul_rn(qv[n], invs2[n]);
            slopes(X, D);
            uniform_sides(X, D);
#pragma unroll
            for (int n = 0; n < N; ++n) {
                const float qs = star_at(X[n], D[n], a);
                const float dqs = star_diff(X[n], X[n + 1], D[n], D[n + 1], a);
                qv[n] = uniform_update(qv[n], c, qs, dss[n], Fs[n], dqs);
            }
        }
        store(rows.out(q), qv);
    }
}

// compute_pressure (SourceEuler.cpp:1345-1376): P alone
__device__ __forceinline__ void pressure_cell(const GeoF &g, const TablesF &t, const PhysF &ph,
                                              const float *__restrict__ S,
                                              const float *__restrict__ E, float *__restrict__ P,
                                              int i, int j)
{
    const int nz = g.nz;
    const size_t c = CELL(i, j);
    if (ph.adiabatic) {
        P[c] = ph.gm1 * E[c];
    } else {
        const float c_s = t.CsIso[i];
        P[c] = S[c] * (c_s * c_s);
    }
}

// velocities from momenta (:498-535), floors; rows 0..nr
template <class Q>
__device__ __forceinline__ void finish_cells(
    const Q &q, const GeoF &g, const TablesF &t, const PhysF &ph, const float *__restrict__ m0,
    const float *__restrict__ m1, const float *__restrict__ m2, const float *__restrict__ m3,
    const float *__restrict__ S_t, const float *__restrict__ E_t,
    const float *__restrict__ vr_in, float *__restrict__ vr_out, float *__restrict__ dv_out,
    float *__restrict__ S_out, float *__restrict__ E_out, const float *__restrict__ Slo_t,
    float *__restrict__ Slo_out, const int *__restrict__ shift, int i)
{
    const int nz = g.nz, nr = g.nr;
    const size_t row = (size_t)i * nz;
    float v[4];
    if (i == nr) {
        q.load(vr_in, row, v);
        q.store(vr_out, row, v);
        return;
    }
    // AdvectSHIFT: the transported cell j of ring k sits at j - shift[k]
    auto at = [&](int ring, int sh, int j) {
        int a = j - sh;
        if (a < 0) a += nz;
        return (size_t)ring * nz + a;
    };
    const int sh = __ldg(shift + i);
    float s[4], sl[4], lo[4], e[4], m2l[4], m3c[4];
#pragma unroll
    QUAD {
        const int j = q.col(k);
        const size_t c = at(i, sh, j), l = at(i, sh, jprev(j, nz));
        s[k] = S_t[c];
        sl[k] = S_t[l];
        m2l[k] = m2[l];
        m3c[k] = m3[c];
        lo[k] = Slo_t[c];
        if (ph.adiabatic) e[k] = E_t[c];
    }
    if (i == 0) {
#pragma unroll
        QUAD v[k] = 0.f;
    } else {
        const int shb = __ldg(shift + i - 1);
        float m0b[4], m1c[4], sb[4];
#pragma unroll
        QUAD {
            const size_t c = at(i, sh, q.col(k)), b = at(i - 1, shb, q.col(k));
            m0b[k] = m0[b];
            m1c[k] = m1[c];
            sb[k] = S_t[b];
        }
#pragma unroll
        QUAD v[k] = __fdiv_rn(m0b[k] + m1c[k], sb[k] + s[k]);
    }
    q.store(vr_out, row, v);
    // the residual angular momenta were formed as sigma (dv Rmed) with the
    // FP32 Rmed of the ring: dividing by that same Rmed returns dv without
    // bias, where multiplying by the FP32 1/Rmed would scale every ring's
    // residual by Rmed 1/Rmed - 1 (up to ~6e-8) in every step, a drift that
    // accumulates over tens of thousands of steps; the divisions are
    // correctly rounded for the same reason
    const float rmed = t.Rmed[i];
#pragma unroll
    QUAD v[k] = __fdiv_rn(m2l[k] + m3c[k], __fmul_rn(sl[k] + s[k], rmed));
    q.store(dv_out, row, v);
#pragma unroll
    QUAD {
        const bool floored = s[k] < ph.sigma_min;
        s[k] = floored ? ph.sigma_min : s[k];
        lo[k] = floored ? 0.f : lo[k];
        if (ph.adiabatic) e[k] = tfloor(e[k], s[k], ph);
    }
    q.store(S_out, row, s);
    q.store(Slo_out, row, lo);
    if (ph.adiabatic) q.store(E_out, row, e);
}

// damping zones (damping.cpp:311-776); block-wide over ring i, part of parts
// blocks that share its columns (the mean kind: one block)
// red: 33 floats, redl: 33 long longs (shared memory)
__device__ __forceinline__ void damp_ring_f(float *X, float *X0, const DampQF &d, int i, int nz,
                                            int outer, float dt, float *red, float *Xlo,
                                            long long *redl, int part, int parts)
{
    const int kind = outer ? d.kind_out : d.kind_in;
    const size_t row = (size_t)i * nz;
    float x0c = 0.f;
    if (kind == 3) {
        const float mean = exact_row_mean(X + row, nz, red, redl);
        if (threadIdx.x == 0) X0[row] = mean;
        x0c = mean;
    } else if (kind == 2) {
        x0c = outer ? d.x0_zero_out[i] : d.x0_zero_in[i];
    }
    const float factor = outer ? d.fac_out[i] : d.fac_in[i];
    const float tau = outer ? d.tau_out : d.tau_in;
    const float ef = __expf(-dt * factor / tau);
    // four loads of each thread in flight
    const int step = blockDim.x * parts;
    for (int j = part * blockDim.x + threadIdx.x; j < nz; j += 4 * step) {
        float x[4], x0[4], lo[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int jj = min(j + k * step, nz - 1);
            x[k] = X[row + jj];
            x0[k] = kind == 1 ? X0[row + jj] : x0c;
            lo[k] = Xlo ? Xlo[row + jj] : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (j + k * step >= nz) break;
            X[row + j + k * step] = (x[k] - x0[k]) * ef + x0[k];
            if (Xlo) Xlo[row + j + k * step] = lo[k] * ef;
        }
    }
    __syncthreads();
}

// fields q0 .. q1 - 1 of ring i (0 v_r, 1 v_phi residual, 2 sigma, 3 energy:
// independent of one another)
__device__ __forceinline__ void damping_ring(const GeoF &g, const DampingF &dm, float dt,
                                             const StateF &s, int i, float *red, long long *redl,
                                             int q0 = 0, int q1 = 4, int part = 0,
                                             int parts = 1)
{
    const int nz = g.nz, nr = g.nr;
    float *X[4] = {s.vr, s.dv, s.sigma, s.energy};
    float *X0[4] = {s.vr0, s.dv0, s.sigma0, s.energy0};
    for (int q = q0; q < q1; ++q) {
        const DampQF &d = dm.q[q];
        const int size = d.vector ? nr + 1 : nr;
        float *lo = q == 2 ? s.sigma_lo : nullptr;
        const bool in = d.kind_in != 0 && d.active_in && i <= d.limit_in;
        const bool out = d.kind_out != 0 && d.active_out && i >= d.limit_out && i < size;
        // a ring mean, the ring's other damping (on a narrow disk the zones
        // overlap) before or after it: one block, or one would read what another
        // writes.  The other kinds leave each column to one thread, inner edge
        // first.
        const bool alone = (in && d.kind_in == 3) || (out && d.kind_out == 3);
        if (alone && part > 0) continue;
        const int p = alone ? 0 : part, of = alone ? 1 : parts;
        if (in) damp_ring_f(X[q], X0[q], d, i, nz, 0, dt, red, lo, redl, p, of);
        if (out) damp_ring_f(X[q], X0[q], d, i, nz, 1, dt, red, lo, redl, p, of);
    }
}

// derived quantities + CFL (SourceEuler.cpp:225-249, cfl.cpp:185-382); block-
// wide over ring i.  mode bits: 1 derived quantities, 2 also c_s, H, T of the
// isothermal disk, 4 CFL minimum into dt_min (float bits, atomicMin)
template <class Q>
__device__ __forceinline__ float derived_cfl_cells(
    const Q &q, const GeoF &g, const TablesF &t, const PhysF &ph, int mode, bool cfl_ring, float md0,
    float vref_frame, const float *__restrict__ S, const float *__restrict__ E,
    const float *__restrict__ vr, const float *__restrict__ dv, const float *__restrict__ qplus,
    const float *__restrict__ qminus, float *__restrict__ cs, float *__restrict__ H,
    float *__restrict__ P, float *__restrict__ T, float *__restrict__ nu,
    const float *__restrict__ corr_phi, const float *__restrict__ corr_r, int i)
{
    const int nz = g.nz;
    const size_t row = (size_t)i * nz;
    float c[4], n[4], e[4], v0[4], v1[4], d0[4], dn[4], qp[4], qm[4];
    if (ph.adiabatic) q.load(E, row, e);
    if (cfl_ring) {
        q.load(vr, row, v0);
        q.load(vr, row + nz, v1);
        q.load(dv, row, d0);
        q.right(dv, row, d0, dn);
        if (ph.adiabatic) {
            q.load(qplus, row, qp);
            q.load(qminus, row, qm);
        }
    }
    if (mode & 1) {
        float sg[4], x[4], h[4];
        q.load(S, row, sg);
        if (ph.adiabatic) {
            const float hfac = t.HFacAdi[i];
            float es[4];
#pragma unroll
            QUAD {
                es[k] = __fdividef(e[k], sg[k]);
                x[k] = ph.c_v_inv * es[k];
                c[k] = sqrtf(ph.g_gm1 * es[k]);
                h[k] = c[k] * hfac;
                n[k] = ph.alpha > 0.f ? ph.alpha * h[k] * c[k] : ph.constant_viscosity;
            }
            q.store(T, row, x);
            q.store(cs, row, c);
            q.store(H, row, h);
#pragma unroll
            QUAD x[k] = ph.gm1 * e[k];
            q.store(P, row, x);
        } else {
            const float c_s = t.CsIso[i], hi = c_s * t.InvOmegaK[i];
            const float ni = ph.alpha > 0.f ? ph.alpha * hi * c_s : ph.constant_viscosity;
#pragma unroll
            QUAD {
                c[k] = c_s;
                h[k] = hi;
                n[k] = ni;
                x[k] = sg[k] * (c_s * c_s);
            }
            q.store(P, row, x);
            if (mode & 2) {
                q.store(cs, row, c);
                q.store(H, row, h);
#pragma unroll
                QUAD x[k] = ph.mu_over_R * x[k] / sg[k];
                q.store(T, row, x);
            }
        }
        q.store(nu, row, n);
    } else {
        q.load(cs, row, c);
        q.load(nu, row, n);
    }
    float local = 3.0e38f;
    if (!cfl_ring) return local;
    const float invcell = t.InvCell[i], invcell2 = t.InvCell2[i], invdrsup = t.InvDiffRsup[i],
                invdxt = t.InvDxTheta[i], invrmed = t.InvRmed[i];
    float cphi[4], cr[4];
    if (ph.stabilize == 2) {
        q.load(corr_phi, row, cphi);
        q.load(corr_r, row, cr);
    }
#pragma unroll
    QUAD {
        const float vres = ph.fast_transport ? d0[k] - md0 : vref_frame + d0[k];
        const float invdt1 = c[k] * invcell;
        const float invdt2 = v0[k] * invdrsup;
        const float invdt3 = vres * invdxt;
        const float dvA = dn[k] - d0[k];
        float invdt4;
        if (ph.art_visc_sn) {
            const float a = fmaxf(v0[k] - v1[k], 0.f) * invdrsup;
            const float b = fmaxf(-dvA, 0.f) * invdxt;
            invdt4 = ph.four_C2 * fmaxf(a, b);
        } else {
            const float eps_pp = __fmul_rn(invrmed, fmaf(dvA, g.invdphi, 0.5f * (v1[k] + v0[k])));
            invdt4 = ph.four_C2 * fmaxf(-fmaf(v1[k] - v0[k], invdrsup, eps_pp), 0.f);
        }
        float invdt5 = 4.f * n[k] * invcell2;
        float invdt6 = 0.f;
        if (ph.adiabatic) invdt6 = ph.inv_hc_limit * fabsf(__fdividef(qp[k] - qm[k], e[k]));
        if (ph.leapfrog) {
            // LeapFrog applies the source terms twice with dt/2 (cfl.cpp:254-317)
            invdt4 *= 0.6f;
            invdt5 *= 0.6f;
            invdt6 *= 0.6f;
        }
        const float s2 = fmaf(
            invdt6, invdt6,
            fmaf(invdt5, invdt5,
                 fmaf(invdt4, invdt4,
                      fmaf(invdt3, invdt3, fmaf(invdt1, invdt1, __fmul_rn(invdt2, invdt2))))));
        float dt_cell = ph.cfl * rsqrtf(s2);
        if (ph.stabilize == 2) {
            // viscous stability limit, cfl.cpp:332-351
            const float cc = fminf(cphi[k], cr[k]);
            if (cc != 0.f) dt_cell = fminf(dt_cell, -ph.cfl / cc);
        }
        local = fminf(local, dt_cell);  // (a cell past the ring's end repeats its last)
    }
    return local;
}

// A ring's mean is formed by its block alone.  The first warp of the disk's ring
// that finishes last takes the shear limits of all pairs of rings and writes the
// disk's step to the host.
__device__ __forceinline__ void derived_cfl_ring(
    const GeoF &g, const TablesF &t, const PhysF &ph, int mode, const float *__restrict__ S,
    const float *__restrict__ E, const float *__restrict__ vr, const float *__restrict__ dv,
    const float *__restrict__ qplus, const float *__restrict__ qminus, float *__restrict__ cs,
    float *__restrict__ H, float *__restrict__ P, float *__restrict__ T, float *__restrict__ nu,
    const CflOut &out, int i, float *red, long long *redl, const float *__restrict__ corr_phi,
    const float *__restrict__ corr_r)
{
    const int nz = g.nz, nr = g.nr;
    const size_t row = (size_t)i * nz;
    const bool do_cfl = (mode & 4) != 0;
    float md0 = 0.f, local = 3.0e38f;
    if (do_cfl) {
        // mean of dv, independent of the block's shape
        md0 = exact_row_mean(dv + row, nz, red, redl);
        if (threadIdx.x == 0) out.mean[i] = md0;
    }
    const bool cfl_ring = do_cfl && i >= 1 && i < nr - 1;
    // standard transport: the ring's frame speed of the Keplerian reference
    const float vref_frame =
        ph.fast_transport ? 0.f : (float)(t.Vref_d[i] - t.Rmed_d[i] * g.omega_frame);
    auto cells = [&](const auto &q) {
        local = fminf(local, derived_cfl_cells(q, g, t, ph, mode, cfl_ring, md0, vref_frame, S, E,
                                               vr, dv, qplus, qminus, cs, H, P, T, nu, corr_phi,
                                               corr_r, i));
    };
    const int bs = blockDim.x, tid = threadIdx.x;
    if (nz % 4 == 0) {
        for (int j = 4 * tid; j < nz; j += 4 * bs) cells(Quad<true>{nz, j, 1});
    } else {
        for (int j = tid; j < nz; j += 4 * bs) cells(Quad<false>{nz, j, bs});
    }
    if (do_cfl) {
        const float m = bmin_f(local, red);
        if (tid >= 32) return;
        unsigned int before = 0;
        if (tid == 0) {
            if (m < 3.0e38f) atomicMin(out.dt_min, __float_as_uint(m));
            __threadfence();
            before = atomicInc(out.done, nr - 1);
        }
        if (__shfl_sync(0xffffffffu, before, 0) != nr - 1u) return;
        __threadfence();
        // shear limit: |vm_i / R_i - vm_{i+1} / R_{i+1}| with vm = Vref + mean dv
        const volatile float *mean = out.mean;
        float shear = 3.0e38f;
        for (int k = tid; k < nr - 1; k += 32) {
            const float denom = fabsf(fmaf(-mean[k + 1], t.InvRmed[k + 1],
                                           fmaf(mean[k], t.InvRmed[k], t.OmRefDiff[k]))) + 1.0e-30f;
            shear = fminf(shear, ph.cfl * g.dphi / denom);
        }
        shear = warp_min_f(shear);
        if (tid == 0) {
            const unsigned int u = __float_as_uint(shear);
            *out.host_dt = __uint_as_float(min(atomicMin(out.dt_min, u), u));
        }
    }
}

}  // namespace fgpu32
