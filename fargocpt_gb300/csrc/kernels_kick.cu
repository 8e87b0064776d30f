// The gas kick of the FP64 form in float-pair arithmetic (fp64_pair.cuh) as
// kernels that march a warp's window of cells through the rings
// (pair_window.cuh).  FP64 is kept for the state updates x += dx and for the
// differences of neighbouring stored values that cancel (v_phi along the ring,
// the pressure), as the pair format carries 2^-48 of each value.
#include "launch.cuh"
#include "kernels.h"
#include "pair_window.cuh"

#include <algorithm>
#include <type_traits>

namespace fgpu {
namespace {

using namespace win;

// The gravitational potential (CalculateNbodyPotential, Pframeforce.cpp:21-86)
// of a central object at the origin without Klahr smoothing (the heliocentric
// frame's usual case; k_potential and k_source_p serve the others) and the
// momentum updates from pressure, potential and centrifugal term
// (update_with_sourceterms, SourceEuler.cpp:325-428).
//
// The central object's distance^2 is R^2 + s^2 (R = Rmed, s = eps H), its
// potential -G m / sqrt(R^2 + s^2) = C (1 + g(u)) with C = -G m / R and, u =
// (s / R)^2, g(u) = (1 + u)^(-1/2) - 1 = -u / (sqrt(1 + u) (1 + sqrt(1 + u))),
// a form without cancellation.  C and its difference between rings come from
// per-ring tables, so the potential's gradient is formed from pairs (the rings'
// difference of C, the differences of the rest) without the rounding of the
// stored FP64 potential, whose gradient cancels about 200 times against
// pressure and centrifugal term.
//
// Bound by the FP32 pipe (59% busy) and issue (57%): 750 instructions per cell
// with three planets, where the two kernels it replaced, one thread per cell,
// took 1294.  2048 x 6144, three planets: 0.476 -> 0.379 ms (0.385 at 4 blocks
// per SM, 0.386 at 6).
template <bool EVEN>
__global__ void __launch_bounds__(kThreads, 5)
    k_source_w(Geo g, Tables t, Phys ph, Bodies b, float2 gm0, float2 dtp, float2 omega_frame,
               int nwin, int chunk, const double *__restrict__ H, const double *__restrict__ S,
               const double *__restrict__ Pr, const double *__restrict__ vr,
               const double *__restrict__ vaz, double *__restrict__ pot,
               double *__restrict__ vr_out, double *__restrict__ vaz_out)
{
    follow_predecessor();
    const int nz = g.nz, nr = g.nr;
    Job job;
    if (!job_of(nwin, nr, chunk, job)) return;
    const Cells<EVEN> c(job.window, nz);
    auto row = [&](int i) { return (size_t)i * nz; };
    const f2x2 pdt = K(dtp);
    const f2x2 cosj = pack(f2{t.cosHi[c.ja], t.cosLo[c.ja]}, f2{t.cosHi[c.jb], t.cosLo[c.jb]});
    const f2x2 sinj = pack(f2{t.sinHi[c.ja], t.sinLo[c.ja]}, f2{t.sinHi[c.jb], t.sinLo[c.jb]});
    const f2x2 one = pack(f2{1.f, 0.f});

    // the potential of row i less C
    auto rest = [&](int i, f2x2 sp) {
        const f2x2 q = sp * T(t, t.InvRmed, i);
        const f2x2 u = q * q;
        const f2x2 w = one + u;
        const f2x2 sq = w * f2_rsqrt(w);
        const f2x2 star = -(K(gm0) * T(t, t.InvRmed, i) * (u / (sq * (one + sq))));
        const f2x2 rm = T(t, t.Rmed, i);
        const f2x2 xc = rm * cosj, yc = rm * sinj, s2 = sp * sp;
        f2x2 acc = star - (K(b.pk_ix) * xc + K(b.pk_iy) * yc);
#pragma unroll 1
        for (int k = 1; k < b.n; ++k) {
            const f2x2 dx = xc - pack(f2{b.xh[k], b.xl[k]});
            const f2x2 dy = yc - pack(f2{b.yh[k], b.yl[k]});
            const f2x2 d2 = (dx * dx + dy * dy) + s2;
            const f2x2 inv_d = f2_rsqrt(d2);
            f2x2 term = inv_d * pack(f2{b.gmh[k], b.gml[k]});
            if ((b.klahr >> k) & 1u) {
                // Klahr's cubic inside r_sm (Pframeforce.cpp:57-66): rare, in FP64
                const double r_sm = b.rsm[k];
                const f2x2 dsm = d2 * inv_d;
                const float lim = __fmul_rn(f2_split(r_sm).h, 1.0f + 0x1p-20f);
                auto inside = [&](f2 d, f2 x) {
                    if (!(d.h < lim)) return x;
                    const double d_sm = f2_to_double(d);
                    if (!(d_sm < r_sm)) return x;
                    const double q = d_sm / r_sm;
                    const double fk = q * q * q * q - 2.0 * (q * q * q) + 2.0 * q;
                    return f2_split(f2_to_double(x) * fk);
                };
                term = pack(inside(first(dsm), first(term)), inside(second(dsm), second(term)));
            }
            acc = acc + term;
        }
        return acc;
    };
    // row r's and row r - 1's sigma, pressure, potential less C, and sums of
    // v_phi over the cell and its right neighbour
    f2x2 s_m, q_m, va_m;
    d2 p_m;
    if (job.i0 > 0) {
        const int i = job.i0 - 1;
        s_m = split(c.load(S + row(i)));
        p_m = c.load(Pr + row(i));
        q_m = rest(i, split(c.load(H + row(i))) * K(ph.pk_eps_smooth));
        const f2x2 va = split(c.load(vaz + row(i)));
        va_m = va + right(va);
    } else {
        s_m = q_m = va_m = pack(f2{0.f, 0.f});
        p_m = d2{0.0, 0.0};
    }
#pragma unroll 1
    for (int r = job.i0; r < job.i1; ++r) {
        const d2 p = c.load(Pr + row(r)), va_d = c.load(vaz + row(r)), vr_d = c.load(vr + row(r));
        const f2x2 s = split(c.load(S + row(r)));
        const f2x2 h = split(c.load(H + row(r)));
        if (r + 1 < job.i1) {
            // the next rows come from DRAM: ask L2 for them
            c.prefetch(Pr + row(r + 1));
            c.prefetch(S + row(r + 1));
            c.prefetch(H + row(r + 1));
            c.prefetch(vaz + row(r + 1));
            c.prefetch(vr + row(r + 1));
        }
        const f2x2 q = rest(r, h * K(ph.pk_eps_smooth));
        const double C = b.gm0 * t.InvRmed[r];
        const d2 qd = join(q);
        c.store(pot + row(r), d2{C + qd.a, C + qd.b});
        const f2x2 va = split(va_d), va_sum = va + right(va);
        const bool active = r >= 1 && r < nr - 1;
        d2 va_new = va_d, vr_new = vr_d;
        if (active && r >= 2) {
            const f2x2 idr = T(t, t.InvDiffRmed, r);
            const f2x2 dp = pack(f2_split(p.a - p_m.a), f2_split(p.b - p_m.b));
            const f2x2 grad = sc(dp, 2.0f) / (s + s_m) +
                              (K(gm0) * T(t, t.DInvRmed, r) + (q - q_m));
            const f2x2 vt = sc(va_sum + va_m, 0.25f) + T(t, t.Rinf, r) * K(omega_frame);
            vr_new = upd(vr_d, pdt * (vt * vt * T(t, t.InvRinf, r) - grad * idr));
        }
        if (active) {
            const f2x2 grad = sc(left_difference(p), 2.0f) / (s + left(s)) + (q - left(q));
            va_new = upd(va_d, -(pdt * (grad * T(t, t.InvDxSrc, r))));
        }
        c.store(vr_out + row(r), vr_new);
        c.store(vaz_out + row(r), va_new);
        if (r == nr - 1) c.store(vr_out + row(nr), c.load(vr + row(nr)));
        s_m = s;
        q_m = q;
        va_m = va_sum;
        p_m = p;
    }
}

// exp(x) - 1 for |x| <= 1/64 in pairs: x + x^2/2 + x^3/6 in pair arithmetic,
// the x^4 tail (below 6.0e-8) in FP32 (its rounding below 2^-48)
__device__ __forceinline__ f2x2 expm1_small(f2x2 x)
{
    const f2x2 x2 = x * x;
    const f2x2 x3 = x2 * x;
    auto k = [](float v) { return make_float2(v, v); };
    float2 p = vfma(x.h, k(1.0f / 5040.0f), k(1.0f / 720.0f));
    p = vfma(p, x.h, k(1.0f / 120.0f));
    p = vfma(p, x.h, k(1.0f / 24.0f));
    const f2x2 tail{vmul(vmul(x2.h, x2.h), p), k(0.f)};
    return x + (sc(x2, 0.5f) + (x3 * P(1.0 / 6.0) + tail));
}
__device__ __forceinline__ f2x2 only_negative(f2x2 sign, f2x2 x)
{
    const bool a = sign.h.x < 0.f, b = sign.h.y < 0.f;
    return f2x2{make_float2(a ? x.h.x : 0.f, b ? x.h.y : 0.f),
                make_float2(a ? x.l.x : 0.f, b ? x.l.y : 0.f)};
}

// Compression heating (SourceEuler.cpp:459-493), the artificial viscosity
// (artificial_viscosity.cpp:11-250: SN or TW pressures, their dissipation, the
// velocity updates) and the derived c_s, H, nu of the ideal EOS
// (compute_sound_speed_normal, compute_scale_height_old, update_viscosity).
// Row r's velocity updates take the pressures of rows r - 1 and r, which are
// kept; the velocities go to other buffers (the neighbouring windows and rows
// need the old ones); the pressures are written as pairs.
//
// Bound by issue (59%) and the integer pipe's conversions (56%): 696
// instructions per cell, where the two kernels it replaced took 1098.
// 2048 x 6144: 0.428 -> 0.355 ms (0.361 at 4 blocks per SM).
template <bool EVEN, bool ADIABATIC>
__global__ void __launch_bounds__(kThreads, 5)
    k_artvisc_w(Geo g, Tables t, Phys ph, float2 dtp, int nwin, int chunk,
                const double *__restrict__ S, const double *__restrict__ vr,
                const double *__restrict__ vaz, double *__restrict__ E, double *__restrict__ Qr,
                double *__restrict__ Qp, double *__restrict__ vr_out, double *__restrict__ vaz_out,
                double *__restrict__ cs, double *__restrict__ H, double *__restrict__ nu)
{
    follow_predecessor();
    const int nz = g.nz, nr = g.nr;
    Job job;
    if (!job_of(nwin, nr, chunk, job)) return;
    const Cells<EVEN> c(job.window, nz);
    auto row = [&](int i) { return (size_t)i * nz; };
    const f2x2 pdt = K(dtp), invdphi = K(g.pk_invdphi), third = P(1.0 / 3.0);
    const f2x2 zero = pack(f2{0.f, 0.f});

    // TW's strain components of row i
    auto strain = [&](int i, f2x2 dv_r, f2x2 v_sum, f2x2 dva, f2x2 &err, f2x2 &epp, f2x2 &div) {
        err = dv_r * T(t, t.InvDiffRsup, i);
        epp = T(t, t.InvRmed, i) * (dva * invdphi + sc(v_sum, 0.5f));
        const f2x2 sum = err + epp;
        div = only_negative(sum, sum);
    };
    // the artificial pressures of row i
    auto pressures = [&](int i, f2x2 s, f2x2 dv_r, f2x2 v_sum, f2x2 dva, f2x2 &qr, f2x2 &qp) {
        if (ph.art_visc_sn) {
            const f2x2 k = K(ph.pk_C2) * s;
            qr = only_negative(dv_r, k * (dv_r * dv_r));
            qp = only_negative(dva, k * (dva * dva));
        } else if (ph.art_visc_tw) {
            f2x2 err, epp, div;
            strain(i, dv_r, v_sum, dva, err, epp, div);
            const f2x2 k = -(T(t, t.LSqTW, i) * s * div), d3 = third * div;
            qr = k * (err - d3);
            qp = k * (epp - d3);
        } else {
            qr = qp = zero;
        }
    };
    f2x2 v0, s_m, qr_m, qp_m;
    d2 v0_d;
    s_m = qr_m = qp_m = zero;
    v0_d = c.load(vr + row(job.i0));
    v0 = split(v0_d);
    if (job.i0 > 0) {
        const int i = job.i0 - 1;
        const f2x2 vb = split(c.load(vr + row(i)));
        s_m = split(c.load(S + row(i)));
        pressures(i, s_m, v0 - vb, v0 + vb, right_difference(c.load(vaz + row(i))), qr_m, qp_m);
    }
#pragma unroll 1
    for (int r = job.i0; r < job.i1; ++r) {
        const d2 v1_d = c.load(vr + row(r + 1)), va_d = c.load(vaz + row(r));
        const d2 s_d = c.load(S + row(r));
        d2 e{0.0, 0.0};
        if (ADIABATIC) e = c.load(E + row(r));
        if (r + 1 < job.i1) {
            c.prefetch(vr + row(r + 2));
            c.prefetch(vaz + row(r + 1));
            c.prefetch(S + row(r + 1));
            if (ADIABATIC) c.prefetch(E + row(r + 1));
        }
        const f2x2 v1 = split(v1_d), s = split(s_d);
        const f2x2 dva = right_difference(va_d), dv_r = v1 - v0;
        f2x2 qr, qp;
        pressures(r, s, dv_r, v1 + v0, dva, qr, qp);
        const bool active = r >= 1 && r < nr - 1;
        if (ADIABATIC) {
            f2x2 de = zero;  // the energy's increment beyond the compression factor
            if (r < nr - 1) {
                const f2x2 div_v = (v1 * T(t, t.Rinf, r + 1) - v0 * T(t, t.Rinf, r)) *
                                       T(t, t.InvDiffRsupRb, r) +
                                   dva * invdphi * T(t, t.InvRmed, r);
                const f2x2 x = -(K(ph.pk_gm1) * pdt * div_v);
                de = split(e) * expm1_small(x);
                // shocks: FP64 exp
                if (fabsf(x.h.x) > 0.015625f) {
                    e.a = e.a * exp(f2_to_double(first(x)));
                    de.h.x = de.l.x = 0.f;
                }
                if (fabsf(x.h.y) > 0.015625f) {
                    e.b = e.b * exp(f2_to_double(second(x)));
                    de.h.y = de.l.y = 0.f;
                }
            }
            if (ph.dissipation && active) {
                if (ph.art_visc_sn) {
                    de = de - pdt * (qr * dv_r * T(t, t.InvDiffRsup, r) +
                                     qp * dva * T(t, t.InvDxTheta, r));
                } else if (ph.art_visc_tw) {
                    f2x2 err, epp, div;
                    strain(r, dv_r, v1 + v0, dva, err, epp, div);
                    const f2x2 d = err - epp;
                    de = de - T(t, t.LSqTW, r) * div * s * third *
                                  (err * err + epp * epp + d * d) * pdt;
                }
            }
            e = upd(e, de);
            if (ph.dissipation) e = d2{floor_e(e.a, s_d.a, ph), floor_e(e.b, s_d.b, ph)};
            c.store(E + row(r), e);
            const f2x2 es = K(ph.pk_g_gm1) * (split(e) / s);
            const f2x2 c_s = es * f2_rsqrt(es);
            const f2x2 h = c_s * T(t, t.HFacAdi, r);
            c.store(cs + row(r), join(c_s));
            c.store(H + row(r), join(h));
            c.store(nu + row(r), ph.alpha > 0 ? join(K(ph.pk_alpha) * h * c_s)
                                              : d2{ph.constant_viscosity, ph.constant_viscosity});
        }
        if (ph.art_visc_sn || ph.art_visc_tw) {
            c.store(Qr + row(r), qr);
            c.store(Qp + row(r), qp);
        }
        d2 va_new = va_d, vr_new = v0_d;
        if (active && ph.art_visc_sn) {
            const f2x2 a = sc(pdt, 2.0f) / (s + left(s));
            va_new = upd(va_d, -(a * (qp - left(qp)) * T(t, t.InvDxTheta, r)));
            if (r >= 2) {
                const f2x2 ar = sc(pdt, 2.0f) / (s + s_m);
                vr_new = upd(v0_d, -(ar * (qr - qr_m) * T(t, t.InvDiffRmed, r)));
            }
        }
        if (active && ph.art_visc_tw) {
            const f2x2 avg = sc(s + left(s), 0.5f);
            va_new = upd(va_d, pdt / avg * T(t, t.InvDxSrc, r) * (qp - left(qp)));
            if (r >= 2) {
                const f2x2 avr = sc(s + s_m, 0.5f);
                const f2x2 br = (qr * T(t, t.Rmed, r) - qr_m * T(t, t.Rmed, r - 1)) -
                                sc(qp + qp_m, 0.5f) * T(t, t.DiffRmed, r);
                vr_new = upd(v0_d, K(ph.pk_rvf) * (pdt / avr) * T(t, t.TwoOverDRmed2, r) * br);
            }
        }
        c.store(vaz_out + row(r), va_new);
        c.store(vr_out + row(r), vr_new);
        if (r == nr - 1) c.store(vr_out + row(nr), v1_d);
        v0 = v1;
        v0_d = v1_d;
        s_m = s;
        qr_m = qr;
        qp_m = qp;
    }
}

// The viscous stress tensor (viscosity.cpp:60-247), the viscous velocity
// update (:249-348 without StabilizeViscosity 1, which the FP64 kernel serves)
// and SubStep3: thermal relaxation (SourceEuler.cpp:632-690), viscous heating
// (:496-536), the radiative alpha factor (:905-912) and the energy update.
// mode bit 1: velocities, bit 2: heating and cooling rates, bit 4: energy.
//
// Row r's update takes tau_r_phi of rows r and r + 1 and the other components
// of rows r - 1 and r: the march forms row r + 1's tau_r_phi and row r's other
// components and keeps row r - 1's.  The velocities go to other buffers (the
// stress of the neighbouring rows and windows needs the old ones); the stress
// tensor and div v are written as pairs (join_pair_fields turns them into
// doubles before a host reads them).
//
// Bound by issue (50%) at 128 registers, 12 warps per SM on average: 1020
// instructions per cell, where the two kernels it replaced took 1875.
// 2048 x 6144: 0.765 -> 0.575 ms (without asking L2 for the rows ahead 0.641; at 96
// registers, 480 bytes of spills, 0.633; at 152 registers 0.678).
template <bool EVEN, bool ADIABATIC>
__global__ void __launch_bounds__(kThreads, 4)
    k_viscous_w(Geo g, Tables t, Phys ph, float2 dtp, float2 beta_inv, int mode, int nwin,
                int chunk, const double *__restrict__ S, const double *__restrict__ nu,
                const double *__restrict__ H, const double *__restrict__ S0,
                const double *__restrict__ E0, const double *__restrict__ vr,
                const double *__restrict__ vaz, double *__restrict__ E, double *__restrict__ divv,
                double *__restrict__ trr, double *__restrict__ tpp, double *__restrict__ trp,
                double *__restrict__ vr_out, double *__restrict__ vaz_out,
                double *__restrict__ qplus, double *__restrict__ qminus)
{
    follow_predecessor();
    const int nz = g.nz, nr = g.nr;
    Job job;
    if (!job_of(nwin, nr, chunk, job)) return;
    const Cells<EVEN> c(job.window, nz);
    auto row = [&](int i) { return (size_t)i * nz; };
    const f2x2 pdt = K(dtp), invdphi = K(g.pk_invdphi), third = P(1.0 / 3.0);
    const f2x2 zero = pack(f2{0.f, 0.f});

    // row r: sigma, nu, v_phi and v_r (doubles and pairs), and the sums of
    // sigma and nu over the cell and its left neighbour
    f2x2 s, n, va, v0, s_sum, n_sum;
    d2 va_d, v0_d;
    // row r's tau_r_phi, row r - 1's sigma, tau_r_r and tau_phi_phi
    f2x2 t_rp, s_m, t_rr_m, t_pp_m;

    // the components at the cell centres of row i, from v_r of its upper face
    auto centred = [&](int i, f2x2 v1, f2x2 &dv, f2x2 &rr, f2x2 &pp) {
        const f2x2 irm = T(t, t.InvRmed, i);
        const f2x2 dphi_v = right_difference(va_d) * invdphi * irm;
        dv = (v1 * T(t, t.Rinf, i + 1) - v0 * T(t, t.Rinf, i)) * T(t, t.InvDiffRsupRb, i) + dphi_v;
        const f2x2 two_n_s = sc(n * s, 2.0f), dv3 = third * dv;
        rr = two_n_s * ((v1 - v0) * T(t, t.InvDiffRsup, i) - dv3);
        pp = two_n_s * ((dphi_v + sc(v1 + v0, 0.5f) * irm) - dv3);
    };
    // tau_r_phi at the lower face of row i from its sums and those of the row
    // below
    auto shear = [&](int i, f2x2 va_i, f2x2 va_b, f2x2 v_i, f2x2 ns_i, f2x2 ns_b, f2x2 ss_i,
                     f2x2 ss_b) {
        const f2x2 dvazirdr =
            (va_i * T(t, t.InvRmed, i) - va_b * T(t, t.InvRmed, i - 1)) * T(t, t.InvDiffRmed, i);
        const f2x2 dvrdphi = (v_i - left(v_i)) * invdphi;
        const f2x2 drp = T(t, t.Rinf, i) * dvazirdr + dvrdphi * T(t, t.InvRinf, i);
        return sc(ns_i + ns_b, 0.25f) * sc(ss_i + ss_b, 0.25f) * drp;
    };
    auto load_row = [&](int i) {
        s = split(c.load(S + row(i)));
        n = split(c.load(nu + row(i)));
        va_d = c.load(vaz + row(i));
        v0_d = c.load(vr + row(i));
        va = split(va_d);
        v0 = split(v0_d);
        s_sum = s + left(s);
        n_sum = n + left(n);
    };

    t_rp = s_m = t_rr_m = t_pp_m = zero;
    if (job.i0 > 0) {
        // row i0 - 1, whose components row i0 takes
        load_row(job.i0 - 1);
        const f2x2 va_b = va, ns_b = n_sum, ss_b = s_sum;
        f2x2 dv;
        centred(job.i0 - 1, split(c.load(vr + row(job.i0))), dv, t_rr_m, t_pp_m);
        s_m = s;
        load_row(job.i0);
        t_rp = shear(job.i0, va, va_b, v0, n_sum, ns_b, s_sum, ss_b);
    } else {
        load_row(0);
    }
#pragma unroll 1
    for (int r = job.i0; r < job.i1; ++r) {
        // row r + 1 (row nr has v_r only)
        const bool up = r + 1 < nr;
        const d2 v1_d = c.load(vr + row(r + 1));
        const f2x2 v1 = split(v1_d);
        d2 va1_d{0.0, 0.0};
        f2x2 s1 = zero, n1 = zero, va1 = zero, s1_sum = zero, n1_sum = zero, t_rp1 = zero;
        if (up) {
            s1 = split(c.load(S + row(r + 1)));
            n1 = split(c.load(nu + row(r + 1)));
            va1_d = c.load(vaz + row(r + 1));
        }
        if (r + 2 < job.i1) {
            // the rows of the next iterations come from DRAM: ask L2 for them
            c.prefetch(vr + row(r + 2));
            c.prefetch(S + row(r + 2));
            c.prefetch(nu + row(r + 2));
            c.prefetch(vaz + row(r + 2));
            if (ADIABATIC) {
                c.prefetch(E + row(r + 2));
                c.prefetch(H + row(r + 2));
            }
        }
        f2x2 dv, t_rr, t_pp;
        centred(r, v1, dv, t_rr, t_pp);
        c.store(divv + row(r), dv);
        c.store(trr + row(r), t_rr);
        c.store(tpp + row(r), t_pp);
        if (r >= 1) c.store(trp + row(r), t_rp);
        if (up) {
            va1 = split(va1_d);
            s1_sum = s1 + left(s1);
            n1_sum = n1 + left(n1);
            t_rp1 = shear(r + 1, va1, va, v1, n1_sum, n_sum, s1_sum, s_sum);
        }
        const bool active = r >= 1 && r < nr - 1;
        const f2x2 t_rp_right = right(t_rp);
        if (mode & 1) {
            d2 va_new = va_d, vr_new = v0_d;
            if (active) {
                const f2x2 dVp =
                    pdt * T(t, t.InvRmed, r) / sc(s_sum, 0.5f) *
                    (T(t, t.TwoOverDRa2, r) *
                         (T(t, t.RinfSq, r + 1) * t_rp1 - T(t, t.RinfSq, r) * t_rp) +
                     (t_pp - left(t_pp)) * invdphi);
                va_new = upd(va_d, dVp);
            }
            if (active && r >= 2) {
                const f2x2 dVr =
                    pdt / sc(s + s_m, 0.5f) * K(ph.pk_rvf) * T(t, t.TwoOverRmedSum, r) *
                    ((T(t, t.Rmed, r) * t_rr - T(t, t.Rmed, r - 1) * t_rr_m) *
                         T(t, t.InvDiffRmed, r) +
                     (t_rp_right - t_rp) * invdphi - sc(t_pp + t_pp_m, 0.5f));
                vr_new = upd(v0_d, dVr);
            }
            c.store(vaz_out + row(r), va_new);
            c.store(vr_out + row(r), vr_new);
            if (r == nr - 1) c.store(vr_out + row(nr), v1_d);
        }
        if (ADIABATIC && (mode & 6)) {
            f2x2 qp = zero, qm = zero;
            const d2 e = c.load(E + row(r));
            const f2x2 ep = split(e);
            if (active) {
                if (ph.cooling_beta) {
                    f2x2 delta_E = ep;
                    if (ph.beta_ref == 1) {
                        delta_E = delta_E - split(c.load(E0 + row(r))) / split(c.load(S0 + row(r))) * s;
                    } else if (ph.beta_ref == 2) {
                        delta_E = delta_E - T(t, t.EModel, r) * s;
                    } else if (ph.beta_ref == 3) {
                        delta_E = delta_E - s * K(ph.pk_emin_fac);
                    }
                    qm = delta_E * T(t, t.OmegaK, r) * K(beta_inv);
                }
                if (ph.heating_viscous) {
                    const f2x2 rp = sc((t_rp + t_rp1) + (t_rp_right + right(t_rp1)), 0.25f);
                    const f2x2 ns = n * s;
                    f2x2 q = (t_rr * t_rr + sc(rp * rp, 2.0f) + t_pp * t_pp) / sc(ns, 2.0f);
                    q = q + P(2.0 / 9.0) * ns * (dv * dv);
                    qp = q * K(ph.pk_hvf);
                    // no heating where nu is zero
                    if (n.h.x == 0.f) qp.h.x = qp.l.x = 0.f;
                    if (n.h.y == 0.f) qp.h.y = qp.l.y = 0.f;
                }
                const f2x2 x = K(ph.pk_mu_gm1_over_R) / s;
                const f2x2 x2 = x * x;
                const f2x2 one = pack(f2{1.f, 0.f});
                const f2x2 alpha = one + split(c.load(H + row(r))) * K(ph.pk_cool_const) *
                                             (x2 * x2) * (ep * ep * ep);
                qp = qp / alpha;
                qm = qm / alpha;
            }
            const d2 qp_d = join(qp);
            d2 qm_d = join(qm);
            if (mode & 4) {
                const d2 sg = c.load(S + row(r));
                d2 e_new = e;
                if (active) {
                    e_new = upd(e, pdt * (qp - qm));
                    // below 10 sigma floors: TAU_EFF is zero on this path, the
                    // equilibrium energy is 0
                    if (below(sg.a, ph.sigma_floor10)) {
                        qm_d.a = qp_d.a;
                        e_new.a = 0.0;
                    }
                    if (below(sg.b, ph.sigma_floor10)) {
                        qm_d.b = qp_d.b;
                        e_new.b = 0.0;
                    }
                }
                c.store(E + row(r), d2{floor_e(e_new.a, sg.a, ph), floor_e(e_new.b, sg.b, ph)});
            }
            c.store(qplus + row(r), qp_d);
            c.store(qminus + row(r), qm_d);
        }
        // advance
        s_m = s;
        t_rr_m = t_rr;
        t_pp_m = t_pp;
        t_rp = t_rp1;
        s = s1;
        n = n1;
        va = va1;
        va_d = va1_d;
        v0 = v1;
        v0_d = v1_d;
        s_sum = s1_sum;
        n_sum = n1_sum;
    }
}

}  // namespace

// Rings per march: as many as leave the device two rounds of resident warps
// (a march forms a ring or less twice, but a short grid needs its warps), at
// most 16.  Measured, ms of the three kernels per step: 2048 x 6144 with 2, 8 and
// 16 rings 1.551, 1.327, 1.308; 512 x 1536 with 1, 2, 4, 8 rings 0.129, 0.115,
// 0.119, 0.126; 128 x 384 with 1, 2, 4 rings 0.029, 0.032, 0.043.
int win::march_rings(int nr, int nwin)
{
    static const int nsm = [] {
        int dev = 0, n = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1)
            n = 152;
        return n;
    }();
    const long long two_rounds = 2LL * nsm * 16;
    return (int)std::max(1LL, std::min(16LL, (long long)nr * nwin / two_rounds));
}

void launch_source_window(const Launch &L, double dt, double omf, const Bodies &b,
                          const State &s, double *vr_out, double *vaz_out)
{
    const int nwin = windows(L.g.nz), chunk = march_rings(L.g.nr, nwin);
    const int jobs = nwin * ((L.g.nr + chunk - 1) / chunk), per = kThreads / 32;
    auto k = L.g.nz % 2 == 0 ? k_source_w<true> : k_source_w<false>;
    launch(k, (jobs + per - 1) / per, kThreads, 0, L.stream,
        L.g, L.t, L.ph, b, split_pair_host(b.gm0), split_pair_host(dt), split_pair_host(omf), nwin,
        chunk, s.H, s.sigma, s.P, s.vr, s.vaz, s.pot, vr_out, vaz_out);
}

void launch_artvisc_pair(const Launch &L, double dt, const State &s, double *vr_out,
                         double *vaz_out)
{
    const int nwin = windows(L.g.nz), chunk = march_rings(L.g.nr, nwin);
    const int jobs = nwin * ((L.g.nr + chunk - 1) / chunk), per = kThreads / 32;
    auto pick = [&](auto even) {
        return L.ph.adiabatic ? k_artvisc_w<even.value, true> : k_artvisc_w<even.value, false>;
    };
    auto k = L.g.nz % 2 == 0 ? pick(std::true_type{}) : pick(std::false_type{});
    launch(k, (jobs + per - 1) / per, kThreads, 0, L.stream,
        L.g, L.t, L.ph, split_pair_host(dt), nwin, chunk, s.sigma, s.vr, s.vaz, s.energy, s.qr,
        s.qphi, vr_out, vaz_out, s.cs, s.H, s.nu);
}

void launch_viscous_pair(const Launch &L, double dt, double beta_inv, int mode, const State &s,
                         double *vr_out, double *vaz_out)
{
    const int nwin = windows(L.g.nz), chunk = march_rings(L.g.nr, nwin);
    const int jobs = nwin * ((L.g.nr + chunk - 1) / chunk), per = kThreads / 32;
    auto pick = [&](auto even) {
        return L.ph.adiabatic ? k_viscous_w<even.value, true> : k_viscous_w<even.value, false>;
    };
    auto k = L.g.nz % 2 == 0 ? pick(std::true_type{}) : pick(std::false_type{});
    launch(k, (jobs + per - 1) / per, kThreads, 0, L.stream,
        L.g, L.t, L.ph, split_pair_host(dt), split_pair_host(beta_inv), mode, nwin, chunk, s.sigma,
        s.nu, s.H, s.sigma0, s.energy0, s.vr, s.vaz, s.energy, s.divv, s.trr, s.tpp, s.trp, vr_out,
        vaz_out, s.qplus, s.qminus);
}

}  // namespace fgpu
