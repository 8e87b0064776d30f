// Cell kernels of the FP64 form in float-pair arithmetic (fp64_pair.cuh), one
// thread per cell: the velocities rebuilt from the transported momenta, and the
// source terms and the stress tensor of the options the window kernels
// (kernels_kick.cu) do not serve.  Every stored double is split into a pair on
// the integer pipe, the arithmetic is pair arithmetic (48 significant bits,
// errors within a few 2^-47 of the operands), and FP64 is kept for three
// things:
//  * the state: an update x += dx adds the pair increment, joined into a
//    double, to the FP64 value of x, so that a step loses the pair's
//    rounding of the increment, not of the state;
//  * the differences of stored values whose gradient cancels: the potential
//    and the pressure in the source terms (neighbouring values agree to 2 or
//    3 digits, so a pair's 2^-48 of each value would be 2^-40 of their
//    difference; the FP64 difference is exact, as in the reference);
//  * the floors (temperature_floor, the sigma floor), screened in FP32 so
//    that only values near a bound take the FP64 comparison, which then
//    gives the reference's clamped value exactly.
// Each kernel cites the reference function it follows and has the grid and
// the ring ranges of its FP64 counterpart.
#include "launch.cuh"
#include "fp64_pair.cuh"
#include "hydro.cuh"
#include "kernels.h"
#include "pair_window.cuh"

#include <math.h>

#include <algorithm>

namespace fgpu {
namespace {

#define CELL(i, j) ((size_t)(i) * (size_t)nz + (size_t)(j))

__device__ __forceinline__ int nxt(int j, int nz) { return j == nz - 1 ? 0 : j + 1; }
__device__ __forceinline__ int prv(int j, int nz) { return j == 0 ? nz - 1 : j - 1; }

__device__ __forceinline__ f2 operator+(f2 a, f2 b) { return f2_sadd(a, b); }
__device__ __forceinline__ f2 operator-(f2 a, f2 b) { return f2_ssub(a, b); }
__device__ __forceinline__ f2 operator-(f2 a) { return f2_neg(a); }
__device__ __forceinline__ f2 operator*(f2 a, f2 b) { return f2_smul(a, b); }
__device__ __forceinline__ f2 operator/(f2 a, f2 b) { return f2_sdiv(a, b); }

// a stored double, a kernel argument or a literal as a pair
__device__ __forceinline__ f2 P(double x) { return f2_split(x); }
// ring i's value of one of the per-ring tables as a pair
__device__ __forceinline__ f2 T(const Tables &t, const double *tab, int i)
{
    const float2 v = t.ptab[(tab - t.tbase) + i];
    return f2{v.x, v.y};
}
// a constant the host split (split_pair_host)
__device__ __forceinline__ f2 K(float2 v) { return f2{v.x, v.y}; }
// the FP64 difference of two stored values, as a pair
__device__ __forceinline__ f2 D(double a, double b) { return f2_split(a - b); }
// x s for a power of two s (exact)
__device__ __forceinline__ f2 sc(f2 x, float s) { return f2{__fmul_rn(x.h, s), __fmul_rn(x.l, s)}; }
// x + dx: the FP64 value plus the joined pair increment
__device__ __forceinline__ double upd(double x, f2 dx) { return x + f2_to_double(dx); }

// update_with_sourceterms (SourceEuler.cpp:369-450): the momentum updates
// from the pressure gradient, the potential and the centrifugal term
__global__ void k_source_p(Geo g, Tables t, float2 dtp, float2 omega_frame,
                           const double *__restrict__ S, const double *__restrict__ Pr,
                           const double *__restrict__ pot, const double *__restrict__ vr_in,
                           const double *__restrict__ vaz_in, double *__restrict__ vr_out,
                           double *__restrict__ vaz_out)
{
    follow_predecessor();
    const int nz = g.nz, nr = g.nr;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;  // 0 .. nr
    if (j >= nz) return;
    const f2 pdt = K(dtp);
    double vr = vr_in[CELL(i, j)];
    if (i >= 2 && i < nr - 1) {
        const size_t c = CELL(i, j), cm = CELL(i - 1, j);
        const f2 idr = T(t, t.InvDiffRmed, i);
        const f2 gradp = sc(D(Pr[c], Pr[cm]), 2.0f) / (P(S[c]) + P(S[cm])) * idr;
        const f2 gradphi = D(pot[c], pot[cm]) * idr;
        const int jn = nxt(j, nz);
        const f2 vsum = (P(vaz_in[c]) + P(vaz_in[CELL(i, jn)])) +
                        (P(vaz_in[cm]) + P(vaz_in[CELL(i - 1, jn)]));
        const f2 vt = sc(vsum, 0.25f) + T(t, t.Rinf, i) * K(omega_frame);
        const f2 centrifugal = vt * vt * T(t, t.InvRinf, i);
        vr = upd(vr, pdt * (centrifugal - (gradp + gradphi)));
    }
    vr_out[CELL(i, j)] = vr;
    if (i < nr) {
        double va = vaz_in[CELL(i, j)];
        if (i >= 1 && i < nr - 1) {
            const size_t c = CELL(i, j), cp = CELL(i, prv(j, nz));
            const f2 invdx = T(t, t.InvDxSrc, i);
            const f2 gradp = sc(D(Pr[c], Pr[cp]), 2.0f) / (P(S[c]) + P(S[cp])) * invdx;
            const f2 gradphi = D(pot[c], pot[cp]) * invdx;
            va = upd(va, -(pdt * (gradp + gradphi)));
        }
        vaz_out[CELL(i, j)] = va;
    }
}

// the viscous stress tensor (viscosity.cpp:60-247) as doubles, as k_stress:
// for StabilizeViscosity 1, whose velocity update is the FP64 kernel's
__global__ void k_stress_p(Geo g, Tables t, const double *__restrict__ S,
                           const double *__restrict__ vr, const double *__restrict__ vaz,
                           const double *__restrict__ nu, double *__restrict__ divv,
                           double *__restrict__ trr, double *__restrict__ tpp,
                           double *__restrict__ trp)
{
    follow_predecessor();
    const int nz = g.nz;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;  // 0 .. nr - 1
    if (j >= nz) return;
    const size_t c = CELL(i, j);
    const int jn = nxt(j, nz);
    const f2 vr0 = P(vr[c]), vr1 = P(vr[CELL(i + 1, j)]);
    const double va0d = vaz[c];
    // v_phi of neighbouring cells of a ring agree to many digits (the orbital
    // speed cancels): their FP64 difference, exact as in the reference
    const f2 dva = D(vaz[CELL(i, jn)], va0d);
    const f2 n = P(nu[c]), sg = P(S[c]);
    const f2 invdphi = K(g.pk_invdphi);
    const f2 irm = T(t, t.InvRmed, i);
    const f2 third = P(1.0 / 3.0);
    const f2 dv = (vr1 * T(t, t.Rinf, i + 1) - vr0 * T(t, t.Rinf, i)) * T(t, t.InvDiffRsupRb, i) +
                  dva * invdphi * irm;
    divv[c] = f2_to_double(dv);
    const f2 two_n_sg = sc(n * sg, 2.0f);
    const f2 drr = (vr1 - vr0) * T(t, t.InvDiffRsup, i);
    trr[c] = f2_to_double(two_n_sg * (drr - third * dv));
    const f2 dpp = dva * invdphi * irm + sc(vr1 + vr0, 0.5f) * irm;
    tpp[c] = f2_to_double(two_n_sg * (dpp - third * dv));
    if (i >= 1) {
        const int jp = prv(j, nz);
        const size_t cm = CELL(i - 1, j), cp = CELL(i, jp), cmp = CELL(i - 1, jp);
        const f2 dvazirdr = (P(va0d) * irm - P(vaz[cm]) * T(t, t.InvRmed, i - 1)) *
                            T(t, t.InvDiffRmed, i);
        const f2 dvrdphi = (vr0 - P(vr[cp])) * invdphi;
        const f2 drp = T(t, t.Rinf, i) * dvazirdr + dvrdphi * T(t, t.InvRinf, i);
        const f2 n4 = sc((n + P(nu[cm])) + (P(nu[cp]) + P(nu[cmp])), 0.25f);
        const f2 s4 = sc((sg + P(S[cm])) + (P(S[cp]) + P(S[cmp])), 0.25f);
        trp[c] = f2_to_double(n4 * s4 * drp);
    }
}

// compute_velocities_from_momenta (TransportEuler.cpp:498-535), the sigma
// floor (SourceEuler.cpp:102-134) and the temperature floor, as k_finish,
// with the azimuthal transport's AdvectSHIFT (:238-268): the transported
// fields of ring i are read at j - its shift; the momenta are pairs
__global__ void k_finish_p(Geo g, Tables t, Phys ph, float2 omf, const f2 *__restrict__ mom0,
                           const f2 *__restrict__ mom1, const f2 *__restrict__ mom2,
                           const f2 *__restrict__ mom3, const double *__restrict__ S_t,
                           const double *__restrict__ E_t, const double *__restrict__ vr_in,
                           double *__restrict__ vr_out, double *__restrict__ vaz_out,
                           double *__restrict__ S_out, double *__restrict__ E_out,
                           const RingPhase *__restrict__ phase)
{
    follow_predecessor();
    const int nz = g.nz, nr = g.nr;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;  // 0 .. nr
    if (j >= nz) return;
    const size_t c = CELL(i, j);
    if (i == nr) {
        vr_out[c] = vr_in[c];
        return;
    }
    // cell j of ring k before the shift
    auto at = [&](int k, int jj) {
        int a = jj - __ldg(&phase[k].shift);
        if (a < 0) a += nz;
        return CELL(k, a);
    };
    const size_t cs = at(i, j);
    const double s = S_t[cs];
    const f2 sp = P(s);
    if (i == 0) {
        vr_out[c] = 0.0;
    } else {
        const size_t cm = at(i - 1, j);
        vr_out[c] = f2_to_double((mom0[cm] + mom1[cs]) / (P(S_t[cm]) + sp));
    }
    const size_t cjm = at(i, prv(j, nz));
    vaz_out[c] = f2_to_double((mom2[cjm] + mom3[cs]) / (P(S_t[cjm]) + sp) *
                                  T(t, t.InvRmed, i) -
                              T(t, t.Rmed, i) * K(omf));
    // s < sigma_min on the bit patterns (sigma_min >= 0; a NaN stays)
    const long long bs = __double_as_longlong(s);
    const bool nan = (bs & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
    const double sf = (!nan && bs < __double_as_longlong(ph.sigma_min)) ? ph.sigma_min : s;
    S_out[c] = sf;
    if (ph.adiabatic) E_out[c] = win::floor_e(E_t[cs], sf, ph);
}

__global__ void k_join_pairs(double *__restrict__ x, size_t n)
{
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x)
        x[k] = f2_to_double(reinterpret_cast<const f2 *>(x)[k]);
}

dim3 grid2(int nz, int rows, int bx) { return dim3((nz + bx - 1) / bx, rows); }

}  // namespace

void launch_source_pair(const Launch &L, double dt, double omf, const double *S, const double *Pr,
                        const double *pot, const double *vr_in, const double *vaz_in,
                        double *vr_out, double *vaz_out)
{
    launch(k_source_p, grid2(L.g.nz, L.g.nr + 1, L.bx), L.bx, 0, L.stream,
        L.g, L.t, split_pair_host(dt), split_pair_host(omf), S, Pr, pot, vr_in, vaz_in, vr_out,
        vaz_out);
}

void launch_stress_pair(const Launch &L, const double *S, const double *vr, const double *vaz,
                        const double *nu, double *divv, double *trr, double *tpp, double *trp)
{
    launch(k_stress_p, grid2(L.g.nz, L.g.nr, L.bx), L.bx, 0, L.stream, L.g, L.t, S, vr, vaz, nu, divv,
                                                                   trr, tpp, trp);
}

void launch_join_pairs(cudaStream_t stream, double *x, size_t n)
{
    const unsigned blocks = (unsigned)std::min<size_t>((n + 255) / 256, 8192);
    k_join_pairs<<<blocks, 256, 0, stream>>>(x, n);
}

void launch_finish_pair(const Launch &L, double omf, double *const mom[4], const double *S_t,
                        const double *E_t, const double *vr_in, double *vr_out, double *vaz_out,
                        double *S_out, double *E_out, const RingPhase *phase)
{
    auto m = [&](int q) { return reinterpret_cast<const f2 *>(mom[q]); };
    launch(k_finish_p, grid2(L.g.nz, L.g.nr + 1, L.bx), L.bx, 0, L.stream,
        L.g, L.t, L.ph, split_pair_host(omf), m(0), m(1), m(2), m(3), S_t, E_t, vr_in,
        vr_out, vaz_out,
        S_out, E_out, phase);
}

}  // namespace fgpu
