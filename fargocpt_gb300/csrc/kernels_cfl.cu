// The derived quantities (recalculate_derived_disk_quantities,
// SourceEuler.cpp:225-249) and the CFL time step (cfl::condition_cfl,
// cfl.cpp:185-382) of the FP64 form in float-pair arithmetic, as a kernel that
// marches windows of cells through the rings (pair_window.cuh).  The ring means
// of v_phi come from the ghost kernel before it, or from k_ring_means.
#include "kernels.h"
#include "launch.cuh"
#include "pair_window.cuh"
#include "reduce.cuh"

#include <algorithm>
#include <type_traits>

namespace fgpu {
namespace {

using namespace win;

__global__ void __launch_bounds__(128) k_ring_means(int nz, const double *__restrict__ vaz,
                                                   double *__restrict__ mean)
{
    follow_predecessor();
    const double m = block_row_mean(vaz + (size_t)blockIdx.x * nz, nz);
    if (threadIdx.x == 0) mean[blockIdx.x] = m;
}

// x truncated to a float, its magnitude at least the smallest normal one (one
// above the floats' range, where pairs overflow too, gives a meaningless float)
__device__ __forceinline__ float trunc_f(double x)
{
    const int w1 = __double2hiint(x);
    const int e = max(w1 & 0x7fffffff, 897 << 20) - (896 << 20);
    const unsigned b = __funnelshift_l((unsigned)__double2loint(x), (unsigned)e, 3);
    return __uint_as_float((b & 0x7fffffffu) | ((unsigned)w1 & 0x80000000u));
}

__device__ __forceinline__ f2x2 larger(f2x2 a, f2x2 b)
{
    const bool x = b.h.x > a.h.x || (b.h.x == a.h.x && b.l.x > a.l.x);
    const bool y = b.h.y > a.h.y || (b.h.y == a.h.y && b.l.y > a.l.y);
    return f2x2{make_float2(x ? b.h.x : a.h.x, y ? b.h.y : a.h.y),
                make_float2(x ? b.l.x : a.l.x, y ? b.l.y : a.l.y)};
}
__device__ __forceinline__ f2x2 positive_part(f2x2 a)
{
    const bool x = a.h.x > 0.f, y = a.h.y > 0.f;
    return f2x2{make_float2(x ? a.h.x : 0.f, y ? a.h.y : 0.f),
                make_float2(x ? a.l.x : 0.f, y ? a.l.y : 0.f)};
}

// A cell's step is CFL over the root of the sum of its six squared inverse
// times (sound speed, radial and azimuthal transport, artificial viscosity,
// viscosity, heating and cooling; LeapFrog's 0.6 on the last three), so the
// disk's is CFL over the root of the largest sum.  Each cell's sum is first
// bounded from above in FP32 (truncated values, differences enlarged by their
// operands' truncation); only rows of a window that may hold a sum above the
// largest found so far (by this warp, or by those that had reported when it
// began: *dt_min) form it in pairs, the differences of v_phi and of Q+ and Q- in
// FP64 (they cancel).  A cell passed over is smaller than one that was formed,
// so the result does not depend on the order.
//
// mode bit 1: derived quantities, bit 2: also those the isothermal disk keeps
// (init), bit 4: CFL.  The grid's first block forms the shear limits that need
// the ghost rings' means; its last block to finish, if host_dt is given,
// writes the step there (page-locked host memory).
//
// Marches of a warp replace one block per ring, which formed every cell's sum in
// pairs, each ring mean twice and the differences' additions on the FP64 pipe
// (that pipe and the issue slots bound it): on 2048 x 6144 cells 0.449 -> 0.205
// ms (its 11 rows of 8 bytes take 0.16 at the memory's rate), on 512 x 1536 0.051
// -> 0.030, on 128 x 384 0.0154 -> 0.0123, the means 0.02 in the ghost kernel;
// 2048 x 6144 with 4, 5, 6 blocks per SM: 0.210, 0.205, 0.213.
template <bool EVEN, bool ADIABATIC>
__global__ void __launch_bounds__(kThreads, 5)
    k_derived_cfl_w(Geo g, Tables t, Phys ph, CflPairs k, int mode, int nwin, int chunk,
                    const double *__restrict__ S, const double *__restrict__ E,
                    const double *__restrict__ vr, const double *__restrict__ vaz,
                    const double *__restrict__ qplus, const double *__restrict__ qminus,
                    double *__restrict__ cs, double *__restrict__ H, double *__restrict__ Pr,
                    double *__restrict__ Te, double *__restrict__ nu,
                    const double *__restrict__ mean, unsigned long long *__restrict__ dt_min,
                    unsigned *__restrict__ done, double *__restrict__ host_dt)
{
    follow_predecessor();
    const int nz = g.nz, nr = g.nr;
    const bool do_cfl = (mode & 4) != 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto row = [&](int i) { return (size_t)i * nz; };
    double shear = 0.0;  // largest |Omega_i - Omega_i+1| of the rings' mean speeds
    f2x2 top = pack(f2{0.f, 0.f});  // largest sum of squares of the lane's cells

    if (blockIdx.x == 0) {
        if (!do_cfl) return;
        const double inner = block_row_mean(vaz, nz);
        const double outer = block_row_mean(vaz + row(nr - 1), nz);
        if (threadIdx.x == 0) {
            const double a = fabs(inner * t.InvRmed[0] - mean[1] * t.InvRmed[1]);
            const double b = fabs(mean[nr - 2] * t.InvRmed[nr - 2] - outer * t.InvRmed[nr - 1]);
            shear = a > b ? a : b;
        }
    } else {
        const int job = (blockIdx.x - 1) * (kThreads / 32) + warp;
        const int ch = job / nwin, window = job - ch * nwin;
        const int i0 = ch * chunk, i1 = min(i0 + chunk, nr);
        const Cells<EVEN> c(window, nz);
        // FP32 bound on the sums worth forming: those not certainly below the
        // step found so far (2^-16 of margin for the roundings)
        const float margin = 1.0f - 0x1p-16f, eps = 0x1p-21f;
        float limit = 0.f;
        d2 v0_d{0.0, 0.0};
        if (do_cfl && i0 < nr) {
            const unsigned long long seen = *(volatile unsigned long long *)dt_min;
            // (a step in the floats' range: not the reset value)
            const unsigned ex = (unsigned)(seen >> 52);
            if (ex > 960u && ex < 1100u) {
                const float r =
                    __fdividef(k.cfl_f, trunc_f(__longlong_as_double((long long)seen)));
                limit = margin * r * r;
            }
            v0_d = c.load(vr + row(i0));
        }
#pragma unroll 1
        for (int r = i0; r < i1; ++r) {
            const bool active = do_cfl && r >= 1 && r < nr - 1;
            f2x2 c_s, n;
            d2 e{0.0, 0.0};
            if (ADIABATIC) e = c.load(E + row(r));
            d2 va{0.0, 0.0}, v1_d{0.0, 0.0}, qp{0.0, 0.0}, qm{0.0, 0.0};
            if (do_cfl) v1_d = c.load(vr + row(r + 1));
            if (active) {
                va = c.load(vaz + row(r));
                if (ADIABATIC) {
                    qp = c.load(qplus + row(r));
                    qm = c.load(qminus + row(r));
                }
            }
            if (mode & 1) {
                const d2 sg = c.load(S + row(r));
                if (r + 1 < i1) {
                    // the next rows come from DRAM: ask L2 for them
                    c.prefetch(S + row(r + 1));
                    if (ADIABATIC) c.prefetch(E + row(r + 1));
                    if (do_cfl) {
                        c.prefetch(vr + row(r + 2));
                        c.prefetch(vaz + row(r + 1));
                        if (ADIABATIC) {
                            c.prefetch(qplus + row(r + 1));
                            c.prefetch(qminus + row(r + 1));
                        }
                    }
                }
                if (ADIABATIC) {
                    const f2x2 es = split(e) / split(sg);
                    c.store(Te + row(r), join(K(k.c_v_inv) * es));
                    const f2x2 c2 = K(ph.pk_g_gm1) * es;
                    c_s = c2 * f2_rsqrt(c2);
                    const f2x2 h = c_s * T(t, t.HFacAdi, r);
                    c.store(cs + row(r), join(c_s));
                    c.store(H + row(r), join(h));
                    c.store(Pr + row(r), d2{ph.gm1 * e.a, ph.gm1 * e.b});
                    if (ph.alpha > 0) {
                        n = K(ph.pk_alpha) * h * c_s;
                        c.store(nu + row(r), join(n));
                    } else {
                        n = K(k.constant_viscosity);
                        c.store(nu + row(r), d2{ph.constant_viscosity, ph.constant_viscosity});
                    }
                } else {
                    const double ci = t.CsIso[r], hi = ci * t.InvOmegaK[r], cc = ci * ci;
                    const double ni = ph.alpha > 0 ? ph.alpha * hi * ci : ph.constant_viscosity;
                    const d2 p{sg.a * cc, sg.b * cc};
                    c.store(Pr + row(r), p);
                    if (mode & 2) {
                        c.store(cs + row(r), d2{ci, ci});
                        c.store(H + row(r), d2{hi, hi});
                        c.store(Te + row(r), d2{ph.mu / ph.Rgas * p.a / sg.a,
                                                ph.mu / ph.Rgas * p.b / sg.b});
                    }
                    c.store(nu + row(r), d2{ni, ni});
                    c_s = T(t, t.CsIso, r);
                    n = pack(f2_split(ni));
                }
            } else {
                c_s = split(c.load(cs + row(r)));
                n = split(c.load(nu + row(r)));
            }
            if (active) {
                const double va_r = __shfl_down_sync(kAll, va.a, 1);  // right of the second
                const double vm = mean[r];
                if (window == 0 && r < nr - 2) {
                    const double d = fabs(vm * t.InvRmed[r] - mean[r + 1] * t.InvRmed[r + 1]);
                    if (d > shear) shear = d;
                }
                // FP32 upper bound of a cell's sum
                auto bound = [&](float cf, float nf, double v0, double v1, double a, double a1,
                                 double p, double m, double en) {
                    auto hi = [&](const double *tab) { return t.ptab[(tab - t.tbase) + r].x; };
                    const float idr = hi(t.InvDiffRsup), idx = hi(t.InvDxTheta);
                    const float f0 = trunc_f(v0), f1 = trunc_f(v1), fa = trunc_f(a),
                                fa1 = trunc_f(a1), fm = trunc_f(vm);
                    const float x1 = cf * hi(t.InvCell), x2 = f0 * idr;
                    const float x3 = ph.fast_transport
                                         ? (fabsf(fa - fm) + eps * (fabsf(fa) + fabsf(fm))) * idx
                                         : fa * idx;
                    const float er = eps * (fabsf(f0) + fabsf(f1)),
                                ea = eps * (fabsf(fa) + fabsf(fa1));
                    float x4;
                    if (ph.art_visc_sn) {
                        x4 = fmaxf((fmaxf(f0 - f1, 0.f) + er) * idr,
                                   (fmaxf(fa - fa1, 0.f) + ea) * idx);
                    } else {
                        x4 = (fabsf(f1 - f0) + er) * idr +
                             hi(t.InvRmed) * ((fabsf(fa1 - fa) + ea) * g.pk_invdphi.x +
                                              0.5f * fabsf(f1 + f0) + er);
                    }
                    x4 *= k.four_C2.x;
                    const float x5 = 4.0f * nf * hi(t.InvCell2);
                    float x6 = 0.f;
                    if (ADIABATIC) {
                        const float fp = trunc_f(p), fq = trunc_f(m);
                        x6 = k.inv_hc.x *
                             __fdividef(fabsf(fp - fq) + eps * (fabsf(fp) + fabsf(fq)),
                                        trunc_f(en));
                    }
                    return (x1 * x1 + x2 * x2 + x3 * x3 + x4 * x4 + x5 * x5 + x6 * x6) *
                           (1.0f + 0x1p-16f);
                };
                const float ba = bound(c_s.h.x, n.h.x, v0_d.a, v1_d.a, va.a, va.b, qp.a, qm.a, e.a);
                const float bb = bound(c_s.h.y, n.h.y, v0_d.b, v1_d.b, va.b, va_r, qp.b, qm.b, e.b);
                // a bound that is not a number is no bound
                const bool need = c.valid > 0 && (!(ba <= limit) || (c.valid > 1 && !(bb <= limit)));
                if (__any_sync(kAll, need)) {
                    const f2x2 idr = T(t, t.InvDiffRsup, r), idx = T(t, t.InvDxTheta, r);
                    const f2x2 v0 = split(v0_d), v1 = split(v1_d);
                    const f2x2 dva = pack(f2_split(va.b - va.a), f2_split(va_r - va.b));
                    const f2x2 x1 = c_s * T(t, t.InvCell, r);
                    const f2x2 x2 = v0 * idr;
                    const f2x2 x3 =
                        (ph.fast_transport ? split(d2{va.a - vm, va.b - vm}) : split(va)) * idx;
                    f2x2 x4;
                    if (ph.art_visc_sn) {
                        x4 = larger(positive_part(v0 - v1) * idr, positive_part(-dva) * idx);
                    } else {
                        const f2x2 epp = T(t, t.InvRmed, r) *
                                         (dva * K(g.pk_invdphi) + sc(v1 + v0, 0.5f));
                        x4 = positive_part(-((v1 - v0) * idr + epp));
                    }
                    x4 = K(k.four_C2) * x4;
                    f2x2 x5 = sc(n * T(t, t.InvCell2, r), 4.0f);
                    f2x2 x6 = pack(f2{0.f, 0.f});
                    if (ADIABATIC)
                        x6 = K(k.inv_hc) * (split(d2{qp.a - qm.a, qp.b - qm.b}) / split(e));
                    if (ph.leapfrog) {
                        x4 = x4 * K(k.leapfrog);
                        x5 = x5 * K(k.leapfrog);
                        x6 = x6 * K(k.leapfrog);
                    }
                    const f2x2 sum = x1 * x1 + x2 * x2 + x3 * x3 + x4 * x4 + x5 * x5 + x6 * x6;
                    const f2x2 m = larger(top, sum);
                    if (c.valid > 0) top.h.x = m.h.x, top.l.x = m.l.x;
                    if (c.valid > 1) top.h.y = m.h.y, top.l.y = m.l.y;
                    const float best = __uint_as_float(__reduce_max_sync(
                        kAll, __float_as_uint(fmaxf(top.h.x, top.h.y))));
                    limit = fmaxf(limit, margin * best);
                }
            }
            v0_d = v1_d;
        }
    }
    if (!do_cfl) return;
    // the warp's step
    f2 best = first(larger(top, f2x2{make_float2(top.h.y, 0.f), make_float2(top.l.y, 0.f)}));
    for (int o = 16; o > 0; o >>= 1) {
        const f2 b{__shfl_down_sync(kAll, best.h, o), __shfl_down_sync(kAll, best.l, o)};
        if (b.h > best.h || (b.h == best.h && b.l > best.l)) best = b;
    }
    if (lane == 0) {
        double d = 1.0e300;
        if (shear > 0.0 || blockIdx.x == 0) d = ph.cfl * g.dphi / (shear + 1.0e-100);
        if (best.h > 0.f) {
            const double dc = f2_to_double(f2_sdiv(f2_split(ph.cfl), f2_sqrt(best)));
            if (dc < d) d = dc;
        }
        if ((blockIdx.x > 0 || warp == 0) && d < 1.0e300)
            atomicMin(dt_min, (unsigned long long)__double_as_longlong(d));
        __threadfence();
    }
    if (!host_dt) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicInc(done, gridDim.x - 1) == gridDim.x - 1) {
            const unsigned long long m = atomicMin(dt_min, ~0ull);
            *host_dt = __longlong_as_double((long long)m);
        }
    }
}

}  // namespace

void launch_ring_means(const Launch &L, const double *vaz, double *mean)
{
    launch(k_ring_means, L.g.nr, 128, 0, L.stream, L.g.nz, vaz, mean);
}

void launch_derived_cfl_pair(const Launch &L, int mode, const State &s, const double *mean,
                             unsigned long long *dt_min, unsigned *done, double *host_dt)
{
    const int nwin = windows(L.g.nz), chunk = march_rings(L.g.nr, nwin);
    const int jobs = nwin * ((L.g.nr + chunk - 1) / chunk), per = kThreads / 32;
    const CflPairs k{split_pair_host(L.ph.four_C2), split_pair_host(L.ph.inv_hc_limit),
                     split_pair_host(0.6), split_pair_host(L.ph.c_v_inv),
                     split_pair_host(L.ph.constant_viscosity), (float)L.ph.cfl};
    auto pick = [&](auto even) {
        return L.ph.adiabatic ? k_derived_cfl_w<even.value, true>
                              : k_derived_cfl_w<even.value, false>;
    };
    auto kernel = L.g.nz % 2 == 0 ? pick(std::true_type{}) : pick(std::false_type{});
    launch(kernel, 1 + (jobs + per - 1) / per, kThreads, 0, L.stream, L.g, L.t, L.ph, k, mode, nwin,
           chunk, s.sigma, s.energy, s.vr, s.vaz, s.qplus, s.qminus, s.cs, s.H, s.P, s.T, s.nu,
           mean, dt_min, done, host_dt);
}

}  // namespace fgpu
