// dsp_device.cuh — shared device-side definitions of the B200 DISORT engine.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/dsp.h"

// Phase markers for cycle-count instrumentation builds; no-ops otherwise.
#ifndef DSP_PHASE_BEGIN
#define DSP_PHASE_BEGIN
#endif
#ifndef DSP_PHASE
#define DSP_PHASE(k)
#endif
#ifndef DSP_PHASE_END
#define DSP_PHASE_END
#endif

namespace dsp {

__host__ __device__ constexpr int pow2ceil(int x) { return x <= 1 ? 1 : 2 * pow2ceil((x + 1) / 2); }
__host__ __device__ constexpr int imax(int a, int b) { return a > b ? a : b; }
__host__ __device__ constexpr int round4(int x) { return (x + 3) & ~3; }

struct DArr {
  const double* p;
  long long s;
  __device__ __forceinline__ double operator()(long long i, long long k = 0) const { return p[i * s + k]; }
  __device__ __forceinline__ const double* row(long long i) const { return p + i * s; }
};

// Constants of the reference's Planck routine, computed on the host with libm
// exactly as Planck.cpp:18-31 does, so the device uses bit-identical values.
struct PlanckConsts {
  double vmax, sigdpi, conc, c1;
};

// Per-stream-count constant tables (host-computed, FluxSolver.cpp:257-290, :126,
// :442-445): mu[N], wt[N], dsim[NN], dinv[NN], ylm[N][N] = P_l(mu_i) at [l*N+i].
struct Tables {
  const double* base;
  __device__ __forceinline__ const double* mu() const { return base; }
};
__host__ __device__ constexpr int tab_mu(int) { return 0; }
__host__ __device__ constexpr int tab_wt(int N) { return N; }
__host__ __device__ constexpr int tab_dsim(int N) { return 2 * N; }
__host__ __device__ constexpr int tab_dinv(int N) { return 2 * N + N / 2; }
__host__ __device__ constexpr int tab_ylm(int N) { return 3 * N; }
__host__ __device__ constexpr int tab_size(int N) { return 3 * N + N * N; }

// Instance record (doubles) written by the setup kernel.
struct InstLayout {
  int hdr, dtau_s, ssa_s, fsc, sig, mode, tau_s, tauc, btr, pkag, yb, stride;
  __host__ __device__ static InstLayout make(int L, int N) {
    InstLayout o;
    o.hdr = 0;
    o.dtau_s = 16;
    o.ssa_s = o.dtau_s + L;
    o.fsc = o.ssa_s + L;
    o.sig = o.fsc + L;
    o.mode = o.sig + L;
    o.tau_s = o.mode + L;
    o.tauc = o.tau_s + L + 1;
    o.btr = o.tauc + L + 1;
    o.pkag = o.btr + L + 1;
    o.yb = o.pkag + L + 1;
    o.stride = round4(o.yb + N + 1);
    return o;
  }
};
// header slots (the general solver also uses H_NAZ .. H_NT)
enum { H_NCUT = 0, H_LYRCUT, H_PTOP, H_PBOT, H_PBOTD, H_DELTAM, H_DMPLUS, H_FBEAM, H_UMU0, H_ALB,
       H_FISOT, H_FISOB, H_NAZ, H_KCONV, H_DONE, H_NT, H_NSLOTS };
static_assert(H_NSLOTS <= 16, "instance header is 16 doubles");

// General-solver instance record: the InstLayout fields for (L, N), then the
// output optical depths utau[NT], their scaled values utaus[NT] and the layer
// of each, lyr[NT] (NT = user taus, or L + 1 levels), and the lowest azimuth mode that
// has no eigensystem and the lowest whose boundary-value problem was singular (the modes
// are solved several at a time; what a mode reports counts once the series reaches it).
struct GenLayout {
  InstLayout il;
  int utau, utaus, lyr, eig, sing, stride;
  __host__ __device__ static GenLayout make(int L, int N, int NT) {
    GenLayout g;
    g.il = InstLayout::make(L, N);
    g.utau = g.il.stride;
    g.utaus = g.utau + NT;
    g.lyr = g.utaus + NT;
    g.eig = g.lyr + NT;
    g.sing = g.eig + 1;
    g.stride = round4(g.sing + 1);
    return g;
  }
};

// Layer record (doubles) written by the layer stage, h = N/2 (rows of HP, h rounded
// up to even, pads zero):
//   X^T [h][HP] | Y^T [h][HP] | k [HP] | E [HP] | F [HP] | beam c, d [HP] each |
//   thermal c, d [HP] each | xr0 | xr1
// (E = exp(-k dtau'), F = 1 - E^2).
// With D = diag(sqrt(w_i mu_i)) and up/down the intensities at the h quadrature
// angles, the layer's modes are phi = D (up + down) = X C, psi = D (up - down) =
// Y D_, where C = E1 a + E2 b + c_p, D_ = E2 b - E1 a + d_p with
// E1 = exp(-k (tau - tau_top)), E2 = exp(-k (tau_bot - tau)); X^T Y = I.  (Row c of
// X^T is mode c.)  The particular solution (c_p, d_p) in these coordinates is
// exp(-tau/mu0) (c, d) for the beam and ((xr0 + xr1 tau) c, xr1 d) for thermal
// emission.  lrec_stride is the space allotted to a record.
__host__ __device__ constexpr int mod_hp(int N) { return N / 2 + ((N / 2) & 1); }
__host__ __device__ constexpr int mod_X(int) { return 0; }
__host__ __device__ constexpr int mod_Y(int N) { return (N / 2) * mod_hp(N); }
__host__ __device__ constexpr int mod_k(int N) { return 2 * (N / 2) * mod_hp(N); }
__host__ __device__ constexpr int mod_E(int N) { return mod_k(N) + mod_hp(N); }
__host__ __device__ constexpr int mod_F(int N) { return mod_k(N) + 2 * mod_hp(N); }
__host__ __device__ constexpr int mod_cb(int N) { return mod_k(N) + 3 * mod_hp(N); }
__host__ __device__ constexpr int mod_db(int N) { return mod_k(N) + 4 * mod_hp(N); }
__host__ __device__ constexpr int mod_ct(int N) { return mod_k(N) + 5 * mod_hp(N); }
__host__ __device__ constexpr int mod_dt(int N) { return mod_k(N) + 6 * mod_hp(N); }
__host__ __device__ constexpr int mod_xr(int N) { return mod_k(N) + 7 * mod_hp(N); }
__host__ __device__ constexpr int mod_size(int N) { return mod_xr(N) + 2; }
__host__ __device__ constexpr int lrec_stride(int N) { return round4(N * N + 4 * N + 2); }
// Boundary-value record (doubles) per layer: H [h][HP] | G [h][HP] | r [HP], and
// in the last solved layer's record the downward intensities at the bottom [HP]
// and the inverse [h][HP] of the surface system.  Before the boundary-value
// kernel runs the area holds the hand-off of a split layer stage.  brec_stride is
// the space allotted to a record.
__host__ __device__ constexpr int brec_H(int) { return 0; }
__host__ __device__ constexpr int brec_G(int N) { return (N / 2) * mod_hp(N); }
__host__ __device__ constexpr int brec_r(int N) { return 2 * (N / 2) * mod_hp(N); }
__host__ __device__ constexpr int brec_dn(int N) { return brec_r(N) + mod_hp(N); }
__host__ __device__ constexpr int brec_inv(int N) { return brec_r(N) + 2 * mod_hp(N); }
__host__ __device__ constexpr int brec_stride(int N) { return round4(N * (2 * N + 2)); }
// Flux solves of few streams keep, instead, per layer what the upward pass needs of it
// (flux_bvp.cuh): W [h][HP] | per stream the constant, the two flux functionals and g
// [h][4] | what the fluxes of the bottom level add to phi [HP] | Planck source at the
// bottom and the top.
__host__ __device__ constexpr int trec_v(int N) { return (N / 2) * mod_hp(N); }
__host__ __device__ constexpr int trec_dphi(int N) { return trec_v(N) + 2 * N; }
__host__ __device__ constexpr int trec_pl(int N) { return trec_dphi(N) + mod_hp(N); }
__host__ __device__ constexpr int trec_stride(int N) { return round4(trec_pl(N) + 2); }
// With Jacobians to follow (flux_jac.cuh): R [h][HP] | per stream what a thermal source's
// value at the top, at the bottom and its slope add to f, then to g [h][6] | inverse of
// the surface system [h][HP] (the last layer's).
__host__ __device__ constexpr int tjac_R(int N) { return trec_stride(N); }
__host__ __device__ constexpr int tjac_s(int N) { return tjac_R(N) + (N / 2) * mod_hp(N); }
__host__ __device__ constexpr int tjac_inv(int N) { return round4(tjac_s(N) + 3 * N); }
__host__ __device__ constexpr int tjac_stride(int N) { return round4(tjac_inv(N) + (N / 2) * mod_hp(N)); }
static_assert(tjac_stride(4) <= brec_stride(4) && tjac_stride(6) <= brec_stride(6) && tjac_stride(16) <= brec_stride(16),
              "Jacobian record");
static_assert(trec_stride(4) <= brec_stride(4) && trec_stride(6) <= brec_stride(6) && trec_stride(16) <= brec_stride(16),
              "transmission record");
static_assert(mod_size(4) <= lrec_stride(4) && mod_size(6) <= lrec_stride(6) && mod_size(14) <= lrec_stride(14) &&
                  mod_size(64) <= lrec_stride(64),
              "layer record");
static_assert(brec_inv(4) + 4 <= brec_stride(4) && brec_inv(6) + 12 <= brec_stride(6) &&
                  brec_inv(64) + 1024 <= brec_stride(64),
              "boundary-value record");

// Pseudo-spherical beam record, per layer: with the layer record's beam slots
// (c0, d0), the beam's particular solution is exp(-xba tau) ((c0, d0) + tau (c1, d1))
// in the layer's modes (computeBeamSourceSpherical, FluxSolver.cpp:650-738;
// :391-419): c1 [h] | d1 [h] | xba | the layer's Chapman factor.
__host__ __device__ constexpr int sph_stride(int N) { return round4(N + 2); }
__host__ __device__ constexpr int sph_xba(int N) { return N; }
__host__ __device__ constexpr int sph_ch(int N) { return N + 1; }

// General-solver layer record: the flux layer record, then the eigenvectors
// and sources at the user polar angles of the current mode:
// GU[numu][N] (columns b[h] | a[h]) | zbu[numu] | z0u[numu] | z1u[numu]
__host__ __device__ constexpr int glrec_gu(int N) { return lrec_stride(N); }
__host__ __device__ constexpr int glrec_stride(int N, int numu) { return round4(lrec_stride(N) + numu * (N + 3)); }

// Per-launch view of a general (DisortSolver) chunk.  Instances are addressed by
// chunk slot ci; ids[ci] is the batch index (inputs, outputs, status).
// A launch covers the modes m .. m + gridDim.y - 1; block row y works on mode m + y,
// with its own copy of the per-mode areas, ms_* doubles apart.
struct GenView {
  int m;                       // first azimuth mode of this launch
  long long ms_layer, ms_bvp, ms_cc, ms_ptab, ms_sph, ms_int;  // per-mode strides
  double* imode;               // per mode and slot: I_m [nt_max][numu]
  int nt_max;                  // output depths per slot in imode
  int numu;                    // user polar angles (0: no intensities)
  int numu_in;                 // num_user_mu of the batch (validated when use_user_mu)
  int nphi, ntau_out, numu_out;
  int user_tau;                // number of user optical depths (0: the L + 1 levels)
  double accur;
  const int* ids;              // [n] batch instance of each slot
  const long long* inst_off;   // [n] instance record offsets (doubles)
  const long long* lay_off;    // [n+1] chunk-local first layer of each slot
  const int* layer_inst;       // [layers] slot of each chunk-local layer
  const int* Ls;               // batch num_layers
  const long long* in_off;     // batch layer_offset (CSR)
  const int* nmoms;            // batch num_phase_func_moments
  const double *dtau, *ssa, *pmom, *temp;  // CSR inputs
  const double* zalt;          // level altitudes, laid out like temp (pseudo-spherical beam only)
  DArr utau, umu, phi, phi0;
  long long lstride;           // layer record stride (glrec_stride)
  double* cc;                  // [layers][N] boundary-value solution of the mode (b[h] | a[h])
  double* ptab;                // per slot: P_l^m(-mu0) [N], then P_l^m(mu_u) [numu][N], of the mode
  double* out_flux[8];         // [batch][ntau_out]
  double* out_int;             // [batch][ntau_out][numu_out][nphi]
  double* out_iavg;            // [batch][ntau_out][numu_out]
  // bidirectional surface (brdf_type != 0): the model's parameters per batch
  // instance, the 200-node azimuth quadrature [gmu | gwt], and per chunk slot
  // the mode's surface table (brdf_stride doubles, written by gen_brdf_kernel)
  int brdf_type;
  DArr brdf_par;
  const double* brdf_q;
  double* brdf;
  // Buras-Emde intensity correction: the tabulated phase function and, per
  // chunk slot, its residual-phase tables (becor_stride doubles)
  int nangles;
  DArr mup;
  const double* phasef;  // [batch layers][nangles], CSR like dtau
  double* becor;
  long long becor_ld;    // doubles per slot: becor_stride of the batch's largest NT
};

// Per-slot tables of the Buras-Emde correction for NT output depths
// (applyNewIntensityCorrection / prepDoubleScatIntegr, DisortSolver.cpp:3568-3640,
// 3812-3876): the residual phase function P''[NT][na], the integration grid
// mu_eq[NT][nf] and its signs [NT][nf], and the normalisation [NT].
constexpr int BE_NF = 100;
__host__ __device__ constexpr long long becor_stride(int NT, int na) {
  return ((long long)NT * (na + 2 * BE_NF + 1) + 3) & ~3ll;
}

// Surface table of one chunk slot for the current azimuth mode
// (computeSurfaceBidir, DisortSolver.cpp:2582-2708): rows r = 0..NN-1 are the
// quadrature angles, r = NN + iu the user polar angles; each row holds
// [beam reflectance | diffuse reflectance of incoming stream 0..NN-1 |
//  directional emissivity (mode 0) | the intensity kernel's reflected-field sum].
// After the rows, kept across the modes: the beam reflectance at each user angle
// for every mode run, [numu][N] (zero for modes not run), which the BRDF
// intensity correction sums (DisortSolver.cpp:306-313, 3783-3787).
__host__ __device__ constexpr int brdf_row(int N) { return N / 2 + 3; }
__host__ __device__ constexpr int brdf_beam_modes(int N, int numu) { return (N / 2 + numu) * brdf_row(N); }
__host__ __device__ constexpr int brdf_stride(int N, int numu) {
  return round4(brdf_beam_modes(N, numu) + numu * N);
}

struct FluxParams {
  int n;          // instances in this launch
  int N, L, pc, nmom;
  uint32_t flags;
  DArr wlo, whi, dtau, ssa, pmom, temp, alb, emis, fbeam, umu0, fisot, fisob, ttop, tbot, zalt, rbot;
  const double* tables;  // tab_* layout for N
  PlanckConsts pk;
  double* inst_rec;
  double* layer_rec;
  double* bvp_rec;
  InstLayout il;
  double* out[8];
  int32_t* status;
  GenView g;  // general-solver launches only
  double* sph = nullptr;      // [n][L][sph_stride], general: [layers][sph_stride] (pseudo-spherical beam only)
};

// The temperature-Jacobian launch of a flux chunk: the vectors r of every degree
// of freedom, per instance [L][h][ndof], and the six outputs [batch][L+1][ndof]
// (already offset to the chunk's first instance).
struct JacView {
  int ndof;         // flux path: L + 2 degrees of freedom (level temperatures 0..L,
                    // surface); general path: the largest L + 2 of the batch
  double* cv;       // [n][L][h][ndof] (general path: [chunk layers][h][ndof])
  double* out[6];   // flux_up, flux_down, mean_intensity, _down, _up, flux_divergence
  int ndof_out;     // general path: column stride of out (>= L + 2 of every instance)
};

// P_l^m(x) for l = m..lmax into y[l * stride] (rows l < m set to 0), the
// recurrence of Legendre.cpp:67-120.  For m > 0 the reference seeds P_m^m with
// the value its previous-mode call left in row m-1; that chain is the product
// below, evaluated in the same order.
__device__ __forceinline__ void legendre_column(int m, double x, int lmax, double* y, int stride) {
  for (int l = 0; l < m && l <= lmax; ++l) y[l * stride] = 0.0;
  if (m == 0) {
    y[0] = 1.0;
    if (lmax >= 1) y[stride] = x;
    double y2 = 1.0, y1 = x;
    for (int l = 2; l <= lmax; ++l) {
      const double v = ((2.0 * l - 1.0) * x * y1 - (l - 1.0) * y2) / l;
      y[l * stride] = v;
      y2 = y1;
      y1 = v;
    }
    return;
  }
  double pmm = 1.0;
  for (int k = 1; k <= m; ++k) pmm = -sqrt((1.0 - 1.0 / (2.0 * k)) * (1.0 - x * x)) * pmm;
  if (m <= lmax) y[m * stride] = pmm;
  const double pm1 = sqrt(2.0 * m + 1.0) * x * pmm;
  if (m + 1 <= lmax) y[(m + 1) * stride] = pm1;
  double y2 = pmm, y1 = pm1;
  for (int l = m + 2; l <= lmax; ++l) {
    const double tmp1 = sqrt(static_cast<double>((l - m) * (l + m)));
    const double tmp2 = sqrt(static_cast<double>((l - m - 1) * (l + m - 1)));
    const double v = ((2.0 * l - 1.0) * x * y1 - tmp2 * y2) / tmp1;
    y[l * stride] = v;
    y2 = y1;
    y1 = v;
  }
}

// Team helpers.  A team is TEAM consecutive threads; TEAM < 32 lives inside a
// warp (synchronised by __syncwarp on its own lanes), TEAM >= 32 is the whole CTA.
template <int TEAM>
__device__ __forceinline__ unsigned team_mask() {
  if constexpr (TEAM >= 32) {
    return 0xffffffffu;
  } else {
    const unsigned lane = threadIdx.x & 31u;
    return ((1u << TEAM) - 1u) << (lane & ~(unsigned)(TEAM - 1));
  }
}

template <int TEAM>
__device__ __forceinline__ void team_sync() {
  if constexpr (TEAM >= 32) {
    __syncthreads();
  } else {
    __syncwarp(team_mask<TEAM>());
  }
}

// 1/x without branches: the hardware approximation (rcp.approx.ftz.f64)
// refined by two Newton-Raphson steps y <- y + y (1 - x y), each about doubling
// the correct bits (Muller et al., Handbook of Floating-Point Arithmetic, 2nd
// ed., section 4.7); within an ulp or two of 1/x for normal x.  Subnormal x
// flush to zero (result +-inf); the pivots it serves are never that small in a
// solvable system.
__device__ __forceinline__ double rcp_newton(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double e = fma(-x, y, 1.0);
  y = fma(y, e, y);
  e = fma(-x, y, 1.0);
  return fma(y, e, y);
}

// Team copies from global to shared memory with 16-byte cp.async (LDGSTS): ROWS
// rows of COLS doubles, contiguous in global memory, LD doubles apart in shared
// memory; and a vector of ND doubles.  COLS, LD and ND even, both ends 16-byte
// aligned (records start on 32 bytes, their parts at even offsets).  Waited for
// with cp_async_wait and made visible to the team by its next barrier.
template <int TEAM, int COLS, int ROWS, int LD>
__device__ __forceinline__ void team_copy_mat(double* dst, const double* src, int t) {
  constexpr int CPR = COLS / 2, CH = ROWS * CPR;
  const unsigned s0 = static_cast<unsigned>(__cvta_generic_to_shared(dst));
#pragma unroll(CH / TEAM <= 8 ? (CH + TEAM - 1) / TEAM : 4)
  for (int k = t; k < CH; k += TEAM) {
    const int r = k / CPR, c2 = k - r * CPR;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s0 + 8u * (unsigned)(r * LD + 2 * c2)),
                 "l"(src + 2 * k)
                 : "memory");
  }
}
template <int TEAM, int ND>
__device__ __forceinline__ void team_copy_vec(double* dst, const double* src, int t) {
  const unsigned s0 = static_cast<unsigned>(__cvta_generic_to_shared(dst));
#pragma unroll(ND / 2 / TEAM <= 8 ? (ND / 2 + TEAM - 1) / TEAM : 4)
  for (int k = t; k < ND / 2; k += TEAM)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s0 + 16u * k), "l"(src + 2 * k) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
// wait until at most N of this thread's most recent groups are pending
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ void set_status(int32_t* status, int i, int code) {
  if (status) atomicMax(status + i, code);
}
// Lowers the mode number in a GenLayout eig or sing slot to m (non-negative doubles
// order like their bit patterns).
constexpr double kNoMode = 1.0e9;
__device__ __forceinline__ void lower_mode(double* slot, int m) {
  atomicMin(reinterpret_cast<long long*>(slot), __double_as_longlong((double)m));
}

}  // namespace dsp
