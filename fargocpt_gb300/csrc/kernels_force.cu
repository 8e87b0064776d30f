// The disk's force on the bodies (ComputeDiskOnPlanetAccel, Force.cpp:23-122) of
// the FP64 form, in float-pair arithmetic (fp64_pair.cuh).
#include "kernels.h"
#include "launch.cuh"
#include "fp64_pair.cuh"
#include "reduce.cuh"

#include <algorithm>


namespace fgpu {
namespace {

constexpr int kForceThreads = 128;

struct ForceBodies {
    int n;           // bodies in this pass (1 .. kForceBodies)
    unsigned klahr;  // bit b: body b has Klahr smoothing (rsm > 0)
    float2 eps;      // ThicknessSmoothing as a pair
    double a[kForceBodies], rsm[kForceBodies];
    float xh[kForceBodies], xl[kForceBodies], yh[kForceBodies], yl[kForceBodies];
};

// Klahr's factor of a cell inside r_sm (Force.cpp:88-100), in FP64
__device__ __noinline__ f2 klahr_weight(f2 w, f2 d2, double rsm)
{
    const double dsm = f2_to_double(f2_mul(d2, f2_rsqrt(d2)));
    if (!(dsm < rsm)) return w;
    const double q = dsm / rsm;
    return f2_split(f2_to_double(w) * -(3.0 * (q * q * q * q) - 4.0 * (q * q * q)));
}

// Up to kForceBodies bodies in one pass over the ring: with CorrectDiskSelfgravity
// the ring mean of sigma is subtracted (Force.cpp:64-66), and the gas mass of the
// ring (gas_total_mass, quantities.cpp:51-74) comes along.  One block per active
// ring writes, for body b, partial[5 b .. 5 b + 4] = (inner x, inner y, outer x,
// outer y, mass) of its ring (split at Rmed < a, the body's distance from the
// origin); k_reduce_cols adds the rings with compensation in a fixed order; G and
// the ring's Surf multiply the ring's sums once.
//
// A lane takes two adjacent cells in packed pairs.  Per body and cell: the
// separation, its smoothed inverse cube and the two products into the sums.  With
// r the hardware's estimate of d^-1 (d^2 the smoothed distance squared) and
// e = 1 - d^2 r^2, |e| < 2^-21, the inverse cube is r^3 (1 - e)^(-3/2) =
// r^3 (1 + 3/2 e + 15/8 e^2 + ...): r^2 and r^3 are error-free products of one
// float, and the series' first two terms end below 2^-60.  Sums and products that
// are only added to others stay unnormalised.
//
// Bound by the FP32 pipe (at 128 threads and 5 blocks per SM; 256 and 3 the same
// on 2048 x 6144 cells, 1% longer on 512 x 1536).  One cell per lane with
// normalised pairs throughout, a Newton step for r, and block sums in FP64: 4
// bodies on 2048 x 6144 cells 0.335 ms; this 0.199.
template <bool EVEN>
__global__ void __launch_bounds__(kForceThreads, 5)
    k_disk_force_bodies(Geo g, Tables t, Phys ph, ForceBodies fb, const double *__restrict__ S,
                        const double *__restrict__ H, double *__restrict__ partial, int width)
{
    follow_predecessor();
    __shared__ double part[kForceThreads / 4], total[8];
    const int nz = g.nz;
    const int i = blockIdx.x + 1;  // radial_first_active .. radial_active_size - 1
    const size_t row = (size_t)i * nz;
    const double mean = block_row_mean(S + row, nz);
    const double m = ph.correct_sg ? mean : 0.0;
    const f2x2 rm = pack(f2{t.RmedHi[i], t.RmedLo[i]});
    const f2x2 eps = pack(f2{fb.eps.x, fb.eps.y});
    // per body, the sums of the x and y terms of the lane's two cells
    f2x2 ax[kForceBodies], ay[kForceBodies];
    float rsm_f[kForceBodies];
#pragma unroll
    for (int b = 0; b < kForceBodies; ++b) {
        ax[b] = ay[b] = pack(f2{0.f, 0.f});
        rsm_f[b] = (float)fb.rsm[b] * (1.0f + 0x1p-18f);
    }
    auto both = [](float a) { return make_float2(a, a); };
    // sum += w d, the product's low part unnormalised
    auto accumulate = [](f2x2 &sum, f2x2 w, f2x2 d) {
        const f2x2 p = two_prod(w.h, d.h);
        const float2 pl = vfma(w.h, d.l, vfma(w.l, d.h, p.l));
        const f2x2 s = two_sum(sum.h, p.h);
        sum = f2x2{s.h, vadd(sum.l, vadd(s.l, pl))};
    };
    for (int j = 2 * threadIdx.x; j < nz; j += 2 * kForceThreads) {
        double sa, sb, ha, hb;
        f2x2 cj, sj;
        if (EVEN) {
            const double2 s = *reinterpret_cast<const double2 *>(S + row + j);
            const double2 h = *reinterpret_cast<const double2 *>(H + row + j);
            sa = s.x, sb = s.y, ha = h.x, hb = h.y;
            cj = f2x2{*reinterpret_cast<const float2 *>(t.cosHi + j),
                      *reinterpret_cast<const float2 *>(t.cosLo + j)};
            sj = f2x2{*reinterpret_cast<const float2 *>(t.sinHi + j),
                      *reinterpret_cast<const float2 *>(t.sinLo + j)};
        } else {
            // the last cell has no second: its sigma is the mean, its terms zero
            const int k = min(j + 1, nz - 1);
            sa = S[row + j], ha = H[row + j], hb = H[row + k];
            sb = j + 1 < nz ? S[row + k] : m;
            cj = f2x2{make_float2(t.cosHi[j], t.cosHi[k]), make_float2(t.cosLo[j], t.cosLo[k])};
            sj = f2x2{make_float2(t.sinHi[j], t.sinHi[k]), make_float2(t.sinLo[j], t.sinLo[k])};
        }
        // sigma less the ring mean: the FP64 difference (they agree closely)
        const f2x2 dsig = pack(f2_split(sa - m), f2_split(sb - m));
        const f2x2 smooth = f2_smul(eps, pack(f2_split(ha), f2_split(hb)));
        const f2x2 s2 = f2_smul(smooth, smooth);
        const f2x2 xc = f2_smul(rm, cj), yc = f2_smul(rm, sj);
#pragma unroll
        for (int b = 0; b < kForceBodies; ++b) {
            if (b < fb.n) {
                const f2x2 dx = f2_ssub(xc, pack(f2{fb.xh[b], fb.xl[b]}));
                const f2x2 dy = f2_ssub(yc, pack(f2{fb.yh[b], fb.yl[b]}));
                // d^2 = s^2 + dx^2 + dy^2
                const f2x2 x2 = two_prod(dx.h, dx.h), y2 = two_prod(dy.h, dy.h);
                const float2 xl = vfma(vadd(dx.h, dx.h), dx.l, x2.l);
                const float2 yl = vfma(vadd(dy.h, dy.h), dy.l, y2.l);
                const f2x2 xy = two_sum(x2.h, y2.h), ds = two_sum(xy.h, s2.h);
                const f2x2 d2 = fast_two_sum(
                    ds.h, vadd(vadd(ds.l, xy.l), vadd(vadd(xl, yl), s2.l)));
                // e = 1 - d^2 r^2, the series' e (3/2 + 15/8 e)
                const float2 r = make_float2(rsqrt_approx(d2.h.x), rsqrt_approx(d2.h.y));
                const f2x2 r2 = two_prod(r, r);
                const float2 mh = vneg(d2.h);
                const float2 e = vfma(vneg(d2.l), r2.h,
                                      vfma(mh, r2.l, vfma(mh, r2.h, both(1.f))));
                const float2 f = vmul(e, vfma(e, both(1.875f), both(1.5f)));
                // w = dsig r^3 (1 + f)
                const f2x2 r3 = two_prod(r2.h, r);
                const float2 r3l = vfma(r2.l, r, r3.l);
                const f2x2 p = two_prod(dsig.h, r3.h);
                const float2 pl = vfma(dsig.h, r3l, vfma(dsig.l, r3.h, p.l));
                f2x2 w = fast_two_sum(p.h, vfma(p.h, f, vfma(pl, f, pl)));
                if ((fb.klahr >> b) & 1u) {
                    // (an FP32 screen passes the cells certainly outside r_sm)
                    if (d2.h.x * r.x < rsm_f[b] || d2.h.y * r.y < rsm_f[b])
                        w = pack(klahr_weight(first(w), first(d2), fb.rsm[b]),
                                 klahr_weight(second(w), second(d2), fb.rsm[b]));
                }
                accumulate(ax[b], w, dx);
                accumulate(ay[b], w, dy);
            }
        }
    }
    f2 v[2 * kForceBodies];
#pragma unroll
    for (int b = 0; b < kForceBodies; ++b) {
        v[2 * b] = pair_halves(ax[b]);
        v[2 * b + 1] = pair_halves(ay[b]);
    }
    block_eight_sums(v, part, total);
    if (threadIdx.x < 2 * fb.n) {
        const int b = threadIdx.x >> 1, c = threadIdx.x & 1;
        const double s = total[threadIdx.x] * (ph.G * t.Surf[i]);
        const bool inner = t.Rmed[i] < fb.a[b];
        double *p = partial + (size_t)blockIdx.x * width + 5 * b;
        p[c] = inner ? s : 0.0;
        p[2 + c] = inner ? 0.0 : s;
        if (c == 0) p[4] = t.Surf[i] * (mean * nz);
    }
}

// the rings' components, one block per component
__global__ void k_reduce_cols(const double *__restrict__ partial, int rows, int width,
                              double *__restrict__ out)
{
    follow_predecessor();
    block_compensated_rows(partial, rows, width, blockIdx.x, out);
}

}  // namespace

void launch_disk_force(const Launch &L, int n, const double *px, const double *py,
                       const double *pa, const double *rsm, const double *S, const double *H,
                       double *partial, double *out)
{
    static_assert(kForceBodies == 4, "the kernel forms eight sums");
    const int rows = L.g.nr - 2;
    auto split = [](double x, float &h, float &l) {
        h = (float)x;
        l = (float)(x - (double)h);
    };
    for (int b0 = 0; b0 < n; b0 += kForceBodies) {
        ForceBodies fb{};
        fb.n = std::min(kForceBodies, n - b0);
        split(L.ph.eps_smooth, fb.eps.x, fb.eps.y);
        for (int b = 0; b < fb.n; ++b) {
            split(px[b0 + b], fb.xh[b], fb.xl[b]);
            split(py[b0 + b], fb.yh[b], fb.yl[b]);
            fb.a[b] = pa[b0 + b];
            fb.rsm[b] = rsm[b0 + b];
            if (fb.rsm[b] > 0.0) fb.klahr |= 1u << b;
        }
        const int width = 5 * fb.n;
        launch(L.g.nz % 2 == 0 ? k_disk_force_bodies<true> : k_disk_force_bodies<false>, rows,
               kForceThreads, 0, L.stream, L.g, L.t, L.ph, fb, S, H, partial, width);
        launch(k_reduce_cols, width, kReduceThreads, 0, L.stream, partial, rows, width,
               out + 5 * b0);
    }
}

}  // namespace fgpu
