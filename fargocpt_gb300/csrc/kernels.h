// Host-side launchers of the FP64 hydro kernels (kernels_fp64.cu).
#pragma once

#include "hydro.cuh"

#include <stddef.h>

// raises a kernel's dynamic shared-memory limit, never lowers it (api.cu)
cudaError_t raise_smem_limit(const void *fn, size_t bytes);

namespace fgpu {

struct Launch {
    Geo g;
    Tables t;
    Phys ph;
    cudaStream_t stream;
    int bx;  // threads per block along the azimuth for cell kernels
    // the kernels' arithmetic in float pairs (kernels_pair.cu and the pair
    // transports) instead of FP64, with FP64 state updates
    bool pair = false;
};

// Constants of one ring's azimuthal passes (pair form), from its mean v_phi
// (ComputeConstantResidual, TransportEuler.cpp:207-236): the velocity the
// residual is about; as pairs k dt, the flux factor dxrad / (Surf k dt), the
// uniform pass's interpolation distance and flux factor (k = 1 / dx for van
// Leer, 1 / (2 dx) for MC: the slopes carry no constant factor); the integer
// shift, in [0, nz); whether the uniform velocity is positive.
struct RingPhase {
    double about;
    float2 kdt, face, au, fu;
    int shift, upwind;
};

void launch_potential(const Launch &L, const Bodies &b, const double *H, double *pot);
void launch_source(const Launch &L, double dt, double omf, const double *S, const double *P,
                   const double *pot, const double *vr_in, const double *vaz_in, double *vr_out,
                   double *vaz_out);
void launch_artvisc_q(const Launch &L, double dt, const double *S, const double *vr,
                      const double *vaz, double *E, double *Qr, double *Qp);
void launch_artvisc_v(const Launch &L, double dt, const double *S, const double *E,
                      const double *Qr, const double *Qp, double *vr, double *vaz, double *cs,
                      double *H, double *nu);
void launch_stress(const Launch &L, const double *S, const double *vr, const double *vaz,
                   const double *nu, double *divv, double *trr, double *tpp, double *trp);
void launch_viscous(const Launch &L, double dt, double beta_inv, int mode, const State &s);
void launch_visc_corr(const Launch &L, const State &s);
// for the CFL kernel that follows (or null): dt_min, reset to a huge step;
// mean, the ring means of v_phi of rings 1 .. nr - 2
void launch_ghost(const Launch &L, const BcSpec &bc, double omf, const State &s,
                  unsigned long long *dt_min, double *mean);
void launch_com_boundary(const Launch &L, const ComSpec &c, const State &s);
void launch_correct_vaz(const Launch &L, double domega, double *vaz);
void launch_cfl_cells(const Launch &L, const State &s, double *out);
void launch_com_damping(const Launch &L, const ComSpec &c, double dt, const State &s);
// rings per radial sweep chunk for this device and disk
int radial_chunk_for(bool pair, bool adiabatic, int nr, int nz);
// pair form: also the ring phases of the azimuthal pass, from vaz
void launch_transport_radial(const Launch &L, double dt, double omf, int chunk, const double *S,
                             const double *vr, const double *vaz, const double *E,
                             double *const mom[4], double *E_out, double *S_out,
                             RingPhase *phase);
// the FP64-arithmetic azimuthal pass, in place (AdvectSHIFT included)
size_t azimuthal_smem_bytes(int nz);
int azimuthal_cells_per_thread(int nz);
cudaError_t prepare_azimuthal(size_t smem);
void launch_transport_azimuthal(const Launch &L, double dt, int block, double *const mom[4],
                                double *E, double *S, const double *vaz, double *ring_ws,
                                size_t smem);
// the float-pair azimuthal pass (kernels_azimuthal.cu): momenta as float
// pairs, into buffers other than its inputs; AdvectSHIFT is left to the
// velocity rebuild
void launch_transport_azimuthal_pair(const Launch &L, double *const mom[4], const double *E,
                                     const double *S, const double *vaz,
                                     double *const mom_out[4], double *E_out, double *S_out,
                                     const RingPhase *phase);
// phase: the azimuthal shifts the pair rebuild applies (pair form)
void launch_finish(const Launch &L, double omf, double *const mom[4], const double *S_t,
                   const double *E_t, const double *vr_in, double *vr_out, double *vaz_out,
                   double *S_out, double *E_out, const RingPhase *phase);
void launch_damping(const Launch &L, const Damping &dm, double dt, const int *rings, int nrings,
                    const State &s);
void launch_derived_cfl(const Launch &L, int mode, const State &s, unsigned long long *dt_min);
void launch_pressure(const Launch &L, const double *S, const double *E, double *P);
// the same cell kernels with their arithmetic in float pairs (kernels_pair.cu);
// the launchers above route to them when L.pair is set
void launch_source_pair(const Launch &L, double dt, double omf, const double *S, const double *Pr,
                        const double *pot, const double *vr_in, const double *vaz_in,
                        double *vr_out, double *vaz_out);
void launch_stress_pair(const Launch &L, const double *S, const double *vr, const double *vaz,
                        const double *nu, double *divv, double *trr, double *tpp, double *trp);
// ring means of v_phi, and the derived quantities and CFL step
// (kernels_cfl.cu; not for StabilizeViscosity 2).  mode: 1 derived quantities, 2
// also the isothermal disk's constant ones, 4 CFL, from the ring means, into
// *dt_min and, if host_dt is given, by the last block to finish (*done counts
// them, zero between launches) into page-locked host memory.
// the CFL kernel of the pair form (StabilizeViscosity 2's limit is the FP64
// kernel's)
inline bool cfl_as_pairs(const Launch &L) { return L.pair && L.ph.stabilize != 2; }
struct CflPairs {
    float2 four_C2, inv_hc, leapfrog, c_v_inv, constant_viscosity;
    float cfl_f;
};
void launch_ring_means(const Launch &L, const double *vaz, double *mean);
void launch_derived_cfl_pair(const Launch &L, int mode, const State &s, const double *mean,
                             unsigned long long *dt_min, unsigned *done, double *host_dt);
// kernels that march windows of cells through the rings (kernels_kick.cu), the
// velocities into vr_out, vaz_out:
// the potential and the momentum source terms, for bodies.star_plain
void launch_source_window(const Launch &L, double dt, double omf, const Bodies &b,
                          const State &s, double *vr_out, double *vaz_out);
// compression heating and artificial viscosity
void launch_artvisc_pair(const Launch &L, double dt, const State &s, double *vr_out,
                         double *vaz_out);
// the stress tensor, the viscous velocity update into vr_out, vaz_out (mode
// bit 1) and SubStep3 (kernels_kick.cu), where stress_as_pairs
void launch_viscous_pair(const Launch &L, double dt, double beta_inv, int mode, const State &s,
                         double *vr_out, double *vaz_out);
// Whether the stress kernel leaves div v and the stress tensor as float pairs
// (hi, lo in the 8 bytes of each double) for the float-pair viscous kernel,
// which reads them so, instead of joined doubles; StabilizeViscosity 1's
// viscous update is the FP64 kernel's, which reads doubles.
inline bool stress_as_pairs(const Launch &L) { return L.pair && L.ph.stabilize != 1; }
// the pairs of n cells joined into doubles in place (div v and the stress
// tensor before they are read as doubles)
void launch_join_pairs(cudaStream_t stream, double *x, size_t n);
void launch_finish_pair(const Launch &L, double omf, double *const mom[4], const double *S_t,
                        const double *E_t, const double *vr_in, double *vr_out, double *vaz_out,
                        double *S_out, double *E_out, const RingPhase *phase);
// bodies one disk-force pass handles
constexpr int kForceBodies = 4;

// the disk force on n bodies (ComputeDiskOnPlanetAccel each) and the gas
// mass: out[5 b .. 5 b + 4] = inner x, inner y, outer x, outer y, mass;
// partial holds 5 min(n, 4) doubles per active ring
void launch_disk_force(const Launch &L, int n, const double *px, const double *py,
                       const double *pa, const double *rsm, const double *S, const double *H,
                       double *partial, double *out);
void launch_gas_quantities(const Launch &L, double radius, double omf, const double *S,
                           const double *vaz, double *partial, double *out);
void launch_scale_sigma(const Launch &L, double *S, double target, const double *mass);
void launch_check_finite(const Launch &L, const double *x, size_t n, unsigned long long *bad);
void launch_accrete(const Launch &L, const AccretionSpec &a, double *S, double *E,
                    const double *vr, const double *vaz, const double *nu, double *out);

}  // namespace fgpu
