// flux_layer.cuh — per-(instance, layer) eigensystems and particular solutions.
//
// Replaces solveEigen (FluxSolver.cpp:459-588), computeBeamSource (:595-643) and
// computeIsotropicSource (:745-831), and interpEigenvec / interpSource of the
// general solver (DisortSolver.cpp:2468-2580).
//
// Eigenproblem: the reference symmetrises (a+b)(a-b) with D = diag(sqrt(w mu)),
// factors -B_s = L L^T and diagonalises S = L^T (-A_s) L (SelfAdjointEigenSolver),
// A_s = D (a+b) D^{-1}, B_s = D (a-b) D^{-1}.  With S = U K^2 U^T the modes of
// phi = D (up + down), psi = D (up - down) are
//   X = L U K^{-1/2},  Y = L^{-T} U K^{1/2},  X^T Y = I,
//   -A_s = Y K Y^T, -B_s = X K X^T, and their inverses X K^{-1} X^T, Y K^{-1} Y^T,
// so the particular solutions are diagonal in them: for thermal emission
// (xr0 + xr1 tau), with v = X^T (D M^{-1} 1), M = diag(mu),
//   c = 2 (1 - w') v / k,  d = c / k;
// for the beam exp(-tau/mu0) with alpha = X^T D M^{-1} (q+ + q-) and
// beta = Y^T D M^{-1} (q+ - q-), q+- the source at the up/down quadrature angles,
//   c = (k alpha - beta/mu0) / (k^2 - mu0^{-2}),
//   d = (k beta - alpha/mu0) / (k^2 - mu0^{-2}).
// U and K are the left singular vectors and values of L^T R, -A_s = R R^T, which a
// one-sided Jacobi iteration finds without forming S: its rotations act on the
// columns of L^T R only (no eigenvector matrix is accumulated), and the small
// singular values keep their relative accuracy.  When -A_s is not positive
// definite (unphysical moments) S is formed, and its eigenvectors are the left singular
// vectors of S + shift I, shifted no further than makes it positive definite; when -B_s
// is not, -A_s = L L^T and S = L^T (-B_s) L give the same modes with the two forms
// exchanged (X = L^{-T} U K^{1/2}, Y = L U K^{-1/2}).
// The quadrature is symmetric (mu_{h+j} = -mu_j, P_l^m(-mu) = (-1)^{l+m} P_l^m(mu)),
// so -B_s holds the phase sums of odd l + m only and -A_s those of even l + m:
//   alpha -/+ beta = M^{-1} (O W - I), M^{-1} (E W - I),
//   O_ij, E_ij = sum_{l + m odd, even} g'_l P_l^m(mu_i) P_l^m(mu_j).
//
// N <= 16: one thread per layer task, every matrix in registers (front kernel,
// then the eigensolver with the record's output); on the flux path, when a schedule
// asks for it, a team of threads per task in shared memory.  N = 32, 64: a team of
// lanes per task, two columns per lane in registers.
#pragma once

#include "dsp_device.cuh"

namespace dsp {

template <int N>
struct LCfg {
  static constexpr int NN = N / 2;
  static_assert(N <= 16, "the team kernel serves N <= 16 on the flux path");
  static constexpr int TEAM = pow2ceil(N);
  static constexpr int CTA = 128;
  static constexpr int TPC = CTA / TEAM;
  static constexpr int NNP = NN + (NN & 1);
  static constexpr int NPAIR = NNP / 2;
  static constexpr int BPT = (NPAIR * NPAIR + TEAM - 1) / TEAM;  // Jacobi 2x2 blocks per thread
  static constexpr int NS = NN + 1;  // padded row stride of NN x NN matrices
  static constexpr int MAT = NN * NS;
  // team shared-memory layout (doubles)
  static constexpr int O_A = 0;            // -A_s, then X
  static constexpr int O_B = O_A + MAT;    // -B_s, then S
  static constexpr int O_L = O_B + MAT;    // Cholesky factor
  static constexpr int O_V = O_L + MAT;    // scratch, then the eigenvectors
  static constexpr int O_T = O_V + MAT;    // scratch, then Y
  static constexpr int O_GL = O_T + MAT;   // g'_l [N]
  static constexpr int O_B1 = O_GL + N;    // beam source sums, D M^{-1} (q+ +/- q-) [NN] each
  static constexpr int O_B2 = O_B1 + NN;
  static constexpr int O_MISC = O_B2 + NN;  // flags
  static constexpr int TEAM_SMEM = round4(O_MISC + 8);
  static constexpr int TAB = tab_ylm(N);   // mu, wt, dsim, dinv; the Legendre table is read through L1
  static constexpr size_t smem_bytes() { return sizeof(double) * (size_t)(TAB + TPC * TEAM_SMEM); }
  // resident CTAs per SM the register budget is sized for: as many as shared
  // memory admits (228 KB, 1 KB reserved per CTA), never below 80 registers
  static constexpr int MINB_SMEM = (int)((228u * 1024u) / (smem_bytes() + 1024u));
  static constexpr int MINB_REGS = 65536 / (CTA * 80);
  static constexpr int MINB = MINB_SMEM < 1 ? 1 : (MINB_SMEM < MINB_REGS ? MINB_SMEM : MINB_REGS);
};

// Whether the layer stage of N streams runs as one thread per task: a thread
// that owns a whole h x h S and its eigenvector matrix in registers runs the
// rotations of a sweep with no shuffles or barriers.
template <int N>
__host__ __device__ constexpr bool layer_split() { return N <= 16; }

// packed lower-triangle index of the symmetric element (r, c)
__host__ __device__ constexpr int tri_idx(int r, int c) {
  return r >= c ? r * (r + 1) / 2 + c : c * (c + 1) / 2 + r;
}

// Hand-off between the two launches of a split layer stage, kept in the
// boundary-value records' area (dead until the boundary-value kernel runs):
// blocks of 32 layer tasks, element e of the block's lane k at
// 32 HS b + e w + k (w = tasks in the block), so that a warp of the
// one-thread-per-task kernels reads or writes an element of 32 tasks in one
// coalesced access.  Per task: flag (0 skipped; 1: L^T R by columns; 2: -A_s is
// indefinite, S = L^T (-A_s) L; 3: -B_s is, L is the factor of -A_s and
// S = L^T (-B_s) L; (S + shift I) / scale in the place of L^T R), the Cholesky factor L
// (packed lower), and with a beam the source vectors D M^{-1} (q+ + q-),
// D M^{-1} (q+ - q-).  Shift and scale of an indefinite task are handed on in its layer
// record, in the place of xr0 and xr1.
template <int NN>
struct Handoff {
  static constexpr int TRI = NN * (NN + 1) / 2;
  static constexpr int S_FLAG = 0, S_F = 1, S_L = S_F + NN * NN, S_B1 = S_L + TRI, S_B2 = S_B1 + NN;
  static constexpr int HS = S_B2 + NN;
};

// Quadrature tables of an N-stream solve passed by value: kernel parameters
// live in the constant bank, so the one-thread-per-task kernels read them as
// uniform operands with compile-time offsets, no loads.
template <int N>
struct ConstTab {
  double mu[N / 2], rmu[N / 2], wt[N / 2], dsim[N / 2], dinv[N / 2];
  double y[N * (N / 2)];  // P_l^m(mu_i), mu_i > 0, at [l * N/2 + i]
};

// ConstTab from a host copy of the tab_* table layout
template <int N>
inline ConstTab<N> make_const_tab(const double* tab) {
  ConstTab<N> c;
  for (int k = 0; k < N / 2; ++k) {
    c.mu[k] = tab[tab_mu(N) + k];
    c.rmu[k] = 1.0 / c.mu[k];
    c.wt[k] = tab[tab_wt(N) + k];
    c.dsim[k] = tab[tab_dsim(N) + k];
    c.dinv[k] = tab[tab_dinv(N) + k];
  }
  for (int l = 0; l < N; ++l)
    for (int k = 0; k < N / 2; ++k) c.y[l * (N / 2) + k] = tab[tab_ylm(N) + l * N + k];
  return c;
}

// address of element e of task j in the lane-interleaved blocks
template <int NN>
__device__ __forceinline__ double* handoff_lane(double* bvp_rec, long long nt, long long j, int e) {
  using H = Handoff<NN>;
  const long long b = j >> 5;
  const long long left = nt - (b << 5);
  const int w = left < 32 ? (int)left : 32;
  return bvp_rec + b * 32 * H::HS + (long long)e * w + (j & 31);
}

// Round-robin pairing of NNP players in round r: (arr[a], arr[NNP-1-a]),
// arr[0] = 0, arr[j] = 1 + (j - 1 + r) mod (NNP - 1).
template <int NNP>
__device__ __forceinline__ int rr_player(int r, int j) {
  int x = j - 1 + r;  // < 2 (NNP - 1) for r < NNP - 1: one conditional subtract replaces the modulo
  if (x >= NNP - 1) x -= NNP - 1;
  return j == 0 ? 0 : 1 + x;
}

// Right-looking Cholesky of the lower triangle of M (NN x NN, stride NS) into Lc,
// row i held by thread i (sub-warp teams): column j's entries are broadcast by
// shuffles.  False if M is not positive definite; every thread leaves through a
// team barrier.
template <int NN, int NS, int TEAM>
__device__ bool team_cholesky_reg(const double* M, double* Lc, int t) {
  static_assert(TEAM <= 32, "shuffle Cholesky needs a sub-warp team");
  const unsigned msk = team_mask<TEAM>();
  double row[NN];
#pragma unroll
  for (int k = 0; k < NN; ++k) row[k] = (t < NN && k <= t) ? M[t * NS + k] : 0.0;
  bool ok = true;
#pragma unroll
  for (int j = 0; j < NN; ++j) {
    const double djj = __shfl_sync(msk, row[j], j, TEAM);
    if (!(djj > 0.0)) ok = false;
    const double ljj = ok ? sqrt(djj) : 1.0;
    const double lij = (t == j) ? ljj : ((t > j && t < NN) ? row[j] / ljj : 0.0);
    if (t < NN) Lc[t * NS + j] = (t >= j) ? lij : 0.0;
#pragma unroll
    for (int k = j + 1; k < NN; ++k) {
      const double lkj = __shfl_sync(msk, lij, k, TEAM);
      if (t >= k && t < NN) row[k] -= lij * lkj;
    }
  }
  if (t < NN)
    for (int k = t + 1; k < NN; ++k) Lc[t * NS + k] = 0.0;
  team_sync<TEAM>();
  return ok;
}

// Whether the Jacobi rotation of pair (p, q) is applied: |apq| above 1e-15 of
// sqrt|app aqq| (about 4.5 ulp).  With the quadratic convergence of cyclic
// Jacobi a threshold at this level rather than 1e-17 saves the last sweep of
// many tasks; an off-diagonal left at that level moves eigenvalues by its square
// and eigenvectors by it over the eigenvalue gap, far below the 1e-9 parity bound.
#ifndef DSP_JACOBI_TOL2
#define DSP_JACOBI_TOL2 1.0e-30
#endif
__device__ __forceinline__ bool jacobi_needed(double apq, double app, double aqq) {
  return fabs(apq) > 1e-300 && apq * apq > DSP_JACOBI_TOL2 * fabs(app * aqq);
}

// Jacobi rotation (Golub & Van Loan, Alg. 8.4.1) zeroing apq; tt = 0 when apq
// is negligible.  t = tan(theta) is the smaller root of t^2 + 2 th t - 1
// with th = d / e, d = aqq - app, e = 2 apq, written as
// t = sgn(th) |e| / (|d| + sqrt(d^2 + e^2)) (one square root, one division).
__device__ __forceinline__ void jacobi_rot(double apq, double app, double aqq, double& c, double& s,
                                           double& tt) {
  c = 1.0;
  s = 0.0;
  tt = 0.0;
  if (jacobi_needed(apq, app, aqq)) {
    const double d = aqq - app, e = 2.0 * apq;
    if (fabs(d) > 1e8 * fabs(e)) {
      tt = e / (2.0 * d);
      c = 1.0 - 0.5 * tt * tt;
    } else {
      const double num = d > 0.0 ? e : (d < 0.0 ? -e : fabs(e));  // sgn(th) |e|, sgn(0) = +1
      tt = num / (fabs(d) + sqrt(d * d + e * e));
      c = rsqrt(tt * tt + 1.0);
    }
    s = tt * c;
  }
}

// One layer task: its instance, layer and addresses.
template <bool GEN>
__device__ __forceinline__ int mode_row() { return GEN ? (int)blockIdx.y : 0; }
template <bool GEN>
__device__ __forceinline__ int mode_of(const FluxParams& p) { return GEN ? p.g.m + (int)blockIdx.y : 0; }

template <int N, bool GEN>
struct LayerTask {
  int i, lc;          // input / status index, layer (top down)
  long long slot;     // instance slot of the launch
  const double* rec;  // instance record
  InstLayout il;
  const double* pml;  // phase-function moments
  double* lrec;       // layer record
  bool live;          // solved in this launch
};
template <int N, bool GEN>
__device__ __forceinline__ LayerTask<N, GEN> layer_task(const FluxParams& p, long long task) {
  LayerTask<N, GEN> q;
  int Lin;
  if constexpr (GEN) {  // ragged layers; task = chunk-local layer
    q.slot = p.g.layer_inst[task];
    q.i = p.g.ids[q.slot];
    q.lc = (int)(task - p.g.lay_off[q.slot]);
    Lin = p.g.Ls[q.i];
    q.il = InstLayout::make(Lin, N);
    q.rec = p.inst_rec + p.g.inst_off[q.slot];
    q.lrec = p.layer_rec + mode_row<GEN>() * p.g.ms_layer + task * p.g.lstride;
    const int lin = (p.flags & DSP_FLAG_INDEX_FROM_BOTTOM) ? Lin - 1 - q.lc : q.lc;
    q.pml = p.g.pmom + (p.g.in_off[q.i] + lin) * (long long)p.pc;
  } else {
    q.i = (int)(task / p.L);
    q.slot = q.i;
    q.lc = (int)(task % p.L);
    q.il = p.il;
    q.rec = p.inst_rec + (long long)q.i * p.il.stride;
    q.lrec = p.layer_rec + task * lrec_stride(N);
    const int lin = (p.flags & DSP_FLAG_INDEX_FROM_BOTTOM) ? p.L - 1 - q.lc : q.lc;
    q.pml = p.pmom.row(q.i) + (long long)lin * p.pc;
  }
  // invalid instances and layers below the absorption cut are not solved; the
  // general solver also skips modes past the instance's last one or after its
  // azimuthal series converged
  q.live = !(p.status && p.status[q.i] == DSP_ERR_INVALID_INPUT) && q.lc < (int)q.rec[H_NCUT];
  if constexpr (GEN) q.live = q.live && mode_of<GEN>(p) <= (int)q.rec[H_NAZ] && q.rec[H_DONE] == 0.0;
  return q;
}
// The general solver's chunk-local record layout of a task's instance.
template <int N>
__device__ __forceinline__ GenLayout task_layout(const FluxParams& p, const LayerTask<N, true>& q) {
  const int L = p.g.Ls[q.i];
  return GenLayout::make(L, N, p.g.user_tau ? p.g.user_tau : L + 1);
}
// Neither -A_s nor -B_s of the task is positive definite: the instance's status; of a
// higher azimuth mode only its entry in the record (the series may end before it).
template <int N, bool GEN>
__device__ __forceinline__ void no_eigensystem(const FluxParams& p, const LayerTask<N, GEN>& q) {
  const int m = mode_of<GEN>(p);
  if constexpr (GEN) lower_mode(const_cast<double*>(q.rec) + task_layout<N>(p, q).eig, m);
  if (m == 0) set_status(p.status, q.i, DSP_ERR_EIGEN);
}
template <bool GEN>
__device__ __forceinline__ long long layer_tasks(const FluxParams& p) {
  if constexpr (GEN) return p.g.lay_off[p.n];
  else return (long long)p.n * p.L;
}
// P_l^m(-mu0) of an instance
template <int N, bool GEN>
__device__ __forceinline__ const double* beam_legendre(const FluxParams& p, const LayerTask<N, GEN>& q) {
  if constexpr (GEN) return p.g.ptab + mode_row<GEN>() * p.g.ms_ptab + q.slot * (long long)(N * (1 + p.g.numu));
  else return q.rec + q.il.yb;
}

// scaled phase coefficient g'_k (disortSet, FluxSolver.cpp:336-386; the general
// solver normalises P_0 to 1, DisortSolver.cpp:669)
template <bool GEN>
__device__ __forceinline__ double phase_coeff(int k, double pk, int mode, double ws, double f, double sig) {
  if (GEN && k == 0) pk = 1.0;
  if (mode == 0) return (2.0 * k + 1.0) * ws * pk;
  if (mode == 1) return (2.0 * k + 1.0) * ws * (pk - f) / (1.0 - f);
  const double kd = (double)k;
  return (2.0 * k + 1.0) * ws * (pk - f * exp(-kd * kd / (2.0 * sig))) / (1.0 - f);
}

// k = sqrt|lambda|, kept off zero: at omega' = 1 one eigenvalue is zero to
// rounding (k ~ 1e-8 either way), and a k below 1e-9 changes no result (the
// solution depends on k^2)
__device__ __forceinline__ double mode_k(double lambda) { return fmax(sqrt(fabs(lambda)), 1e-9); }

// exponent of a layer's E = exp(-k dtau): for a mode of -k (-B_s indefinite) E grows, no
// further than E^2 can be formed (its reciprocal is zero to rounding long before)
__device__ __forceinline__ double mode_exponent(double k, double dtau) { return -fmax(k * dtau, -300.0); }

// the beam's cosine, moved off a resonance mu0 k = 1 (FluxSolver.cpp:610-618)
__device__ __forceinline__ bool beam_resonant(double k, double umu0) {
  return fabs(1.0 - umu0 * umu0 * k * k) < 1000.0 * 2.220446049250313e-16;
}

// thermal source of a layer: intercept and slope in scaled depth (FluxSolver.cpp:745-787)
template <class Q>
__device__ __forceinline__ void thermal_source(const Q& q, double& xr0, double& xr1) {
  const double dts = q.rec[q.il.dtau_s + q.lc], taus_top = q.rec[q.il.tau_s + q.lc];
  const double pk0 = q.rec[q.il.pkag + q.lc], pk1 = q.rec[q.il.pkag + q.lc + 1];
  xr1 = 0.0;
  if (dts > 1e-4) xr1 = (pk1 - pk0) / dts;
  xr0 = pk0 - xr1 * taus_top;
}

// ---------------------------------------------------------------------------
// Layer stage with a team of threads per task, matrices in shared memory.
// ---------------------------------------------------------------------------
template <int N>
__global__ void __launch_bounds__(LCfg<N>::CTA, LCfg<N>::MINB) flux_layer_kernel(FluxParams p) {
  using C = LCfg<N>;
  constexpr int NN = C::NN, TEAM = C::TEAM, NNP = C::NNP, NPAIR = C::NPAIR, NS = C::NS, BPT = C::BPT;
  constexpr int HP = mod_hp(N);
  constexpr int BPA = NPAIR;  // blocks (a, b) per column pair b
  extern __shared__ double smem[];
  // CTA-level constant tables
  for (int k = threadIdx.x; k < C::TAB; k += blockDim.x) smem[k] = p.tables[k];
  __syncthreads();
  const double* mu = smem + tab_mu(N);
  const double* wt = smem + tab_wt(N);
  const double* dsim = smem + tab_dsim(N);
  const double* dinv = smem + tab_dinv(N);
  const double* Y = p.tables + tab_ylm(N);

  const int team = threadIdx.x / TEAM, t = threadIdx.x % TEAM;
  const long long task = (long long)blockIdx.x * C::TPC + team;
  if (task >= layer_tasks<false>(p)) return;
  const LayerTask<N, false> q = layer_task<N, false>(p, task);
  if (!q.live) return;
  double* sm = smem + C::TAB + team * C::TEAM_SMEM;
  double* MA = sm + C::O_A;
  double* MB = sm + C::O_B;
  double* LC = sm + C::O_L;
  double* V = sm + C::O_V;
  double* T = sm + C::O_T;
  double* gl = sm + C::O_GL;
  double* b1 = sm + C::O_B1;
  double* b2 = sm + C::O_B2;
  double* misc = sm + C::O_MISC;
  const double ws = q.rec[q.il.ssa_s + q.lc];
  {
    const int mode = (int)q.rec[q.il.mode + q.lc];
    const double f = q.rec[q.il.fsc + q.lc], sig = q.rec[q.il.sig + q.lc];
    for (int k = t; k < N; k += TEAM) gl[k] = phase_coeff<false>(k, q.pml[k], mode, ws, f, sig);
  }
  team_sync<TEAM>();
  // ---- -A_s and -B_s from the even and odd phase sums ----------------------
  for (int it = t; it < NN * NN; it += TEAM) {
    const int r = it / NN, c = it % NN;
    if (c > r) continue;
    double so = 0.0, se = 0.0;
    for (int l = 0; l < N; l += 2) {
      so += (gl[l + 1] * Y[(l + 1) * N + r]) * Y[(l + 1) * N + c];
      se += (gl[l] * Y[(l) * N + r]) * Y[(l) * N + c];
    }
    const double rm = 1.0 / mu[r], dl = r == c ? rm : 0.0;
    const double vb = -dsim[r] * ((wt[c] * so) * rm - dl) * dinv[c];
    const double va = -dsim[r] * ((wt[c] * se) * rm - dl) * dinv[c];
    MB[r * NS + c] = vb;
    MB[c * NS + r] = vb;
    MA[r * NS + c] = va;
    MA[c * NS + r] = va;
  }
  const double fbeam = q.rec[H_FBEAM];
  const bool beam = fbeam > 0.0;
  if (beam) {
    // (2 - delta_m0) F0 / 4pi sum_k g'_k P_k^m(mu_r) P_k^m(-mu0) by parity (DisortSolver.cpp:1361-1368)
    const double* yb = beam_legendre<N, false>(p, q);
    const double fac = fbeam / (4.0 * 3.14159265358979323846);
    for (int r = t; r < NN; r += TEAM) {
      double so = 0.0, se = 0.0;
      for (int l = 0; l < N; l += 2) {
        so += gl[l + 1] * Y[(l + 1) * N + r] * yb[l + 1];
        se += gl[l] * Y[(l) * N + r] * yb[l];
      }
      const double dm = dsim[r] / mu[r];
      b1[r] = dm * (2.0 * fac * se);
      b2[r] = dm * (2.0 * fac * so);
    }
  }
  team_sync<TEAM>();
  // ---- Cholesky of -B_s, else of -A_s (:521-558) ---------------------------
  bool primary = team_cholesky_reg<NN, NS, TEAM>(MB, LC, t);
  if (!primary && !team_cholesky_reg<NN, NS, TEAM>(MA, LC, t)) {
    if (t == 0) set_status(p.status, q.i, DSP_ERR_EIGEN);
    return;
  }
  // S = L^T M L, M = -A_s (primary) or -B_s (fallback)
  {
    const double* M = primary ? MA : MB;
    for (int it = t; it < NN * NN; it += TEAM) {
      const int r = it / NN, c = it % NN;
      double s = 0.0;
      for (int k = c; k < NN; ++k) s += M[r * NS + k] * LC[k * NS + c];
      T[r * NS + c] = s;
    }
  }
  team_sync<TEAM>();
  for (int it = t; it < NN * NN; it += TEAM) {
    const int r = it / NN, c = it % NN;
    V[r * NS + c] = (r == c) ? 1.0 : 0.0;
    if (c > r) continue;
    double s = 0.0;
    for (int k = r; k < NN; ++k) s += LC[k * NS + r] * T[k * NS + c];
    MB[r * NS + c] = s;
    MB[c * NS + r] = s;
  }
  team_sync<TEAM>();
  double* const Sc = MB;
  double* const Sn = MB;
  // In place: in a round every 2x2 block of S is read and written by its owner
  // only, and the diagonal blocks a rotation is computed from are written by
  // their owner after it has received that rotation.
  for (int sweep = 0; sweep < 20; ++sweep) {
    for (int r = 0; r < NNP - 1; ++r) {
      // rotation of pair a is computed by thread a; each thread then needs the
      // rotations of its block's two pairs only (blocks are assigned statically)
      double c = 1.0, sn = 0.0, tt = 0.0;
      if (t < NPAIR) {
        const int pp = rr_player<NNP>(r, t), qq = rr_player<NNP>(r, NNP - 1 - t);
        if (pp < NN && qq < NN) {
          jacobi_rot(Sc[pp * NS + qq], Sc[pp * NS + pp], Sc[qq * NS + qq], c, sn, tt);
        }
      }
#pragma unroll
      for (int k = 0; k < BPT; ++k) {
        const int blk = t + k * TEAM;
        const bool act = blk < NPAIR * NPAIR;
        const int a = act ? blk / NPAIR : 0, b = act ? blk % NPAIR : 0;  // NPAIR is a power of two or small
        const unsigned m = team_mask<TEAM>();
        const double ca = __shfl_sync(m, c, a, TEAM), sa = __shfl_sync(m, sn, a, TEAM), ta = __shfl_sync(m, tt, a, TEAM);
        const double cb = __shfl_sync(m, c, b, TEAM), sb = __shfl_sync(m, sn, b, TEAM);
        if (!act) continue;
        const int pa = rr_player<NNP>(r, a), qa = rr_player<NNP>(r, NNP - 1 - a);
        const int pb = rr_player<NNP>(r, b), qb = rr_player<NNP>(r, NNP - 1 - b);
        const bool va = qa < NN && pa < NN, vb = qb < NN && pb < NN;
        if (a == b) {
          if (va) {
            const double apq = Sc[pa * NS + qa];
            Sn[pa * NS + pa] = Sc[pa * NS + pa] - ta * apq;
            Sn[qa * NS + qa] = Sc[qa * NS + qa] + ta * apq;
            const double off = (ta != 0.0) ? 0.0 : apq;
            Sn[pa * NS + qa] = off;
            Sn[qa * NS + pa] = off;
          } else {
            const int x = pa < NN ? pa : qa;
            if (x < NN) Sn[x * NS + x] = Sc[x * NS + x];
          }
        } else {
          // rows of pair a (rotated), columns of pair b (rotated); absent
          // (padding) indices act as the identity
          const int ri[2] = {pa, qa}, cj[2] = {pb, qb};
          double X[2][2];
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
              const int rr = ri[u], cc = cj[v];
              X[u][v] = (rr < NN && cc < NN) ? Sc[rr * NS + cc] : 0.0;
            }
          double Y2[2][2];
          if (va) {
#pragma unroll
            for (int v = 0; v < 2; ++v) {
              Y2[0][v] = ca * X[0][v] - sa * X[1][v];
              Y2[1][v] = sa * X[0][v] + ca * X[1][v];
            }
          } else {
#pragma unroll
            for (int v = 0; v < 2; ++v) { Y2[0][v] = X[0][v]; Y2[1][v] = X[1][v]; }
          }
          double Z2[2][2];
          if (vb) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              Z2[u][0] = cb * Y2[u][0] - sb * Y2[u][1];
              Z2[u][1] = sb * Y2[u][0] + cb * Y2[u][1];
            }
          } else {
#pragma unroll
            for (int u = 0; u < 2; ++u) { Z2[u][0] = Y2[u][0]; Z2[u][1] = Y2[u][1]; }
          }
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
              const int rr = ri[u], cc = cj[v];
              if (rr < NN && cc < NN) Sn[rr * NS + cc] = Z2[u][v];
            }
        }
        // eigenvectors V <- V J for pair b: this thread's share of the rows
        if (vb) {
          const int rows_per = (NN + BPA - 1) / BPA;  // blocks sharing pair b split its rows
          const int r0 = a * rows_per;
#pragma unroll 4
          for (int row = r0; row < r0 + rows_per && row < NN; ++row) {
            const double vp = V[row * NS + pb], vq = V[row * NS + qb];
            V[row * NS + pb] = cb * vp - sb * vq;
            V[row * NS + qb] = sb * vp + cb * vq;
          }
        }
      }
      team_sync<TEAM>();
    }
    // stop when a further sweep would rotate no pair (the sweep that finds
    // nothing to do is not run)
    if (t == 0) misc[1] = 0.0;
    team_sync<TEAM>();
    for (int it = t; it < NN * NN; it += TEAM) {
      const int r = it / NN, c = it % NN;
      if (c > r && jacobi_needed(Sc[r * NS + c], Sc[r * NS + r], Sc[c * NS + c])) misc[1] = 1.0;
    }
    team_sync<TEAM>();
    const bool more = misc[1] != 0.0;
    team_sync<TEAM>();
    if (!more) break;
  }
  // ---- modes and particular solutions, one thread per mode ------------------
  for (int c = t; c < NN; c += TEAM) {
    const double k = mode_k(Sc[c * NS + c]);
    // lambda < 0 beyond rounding: M is indefinite, and its inverse carries the sign
    const bool lneg = Sc[c * NS + c] < -1e-10;
    const double sk = sqrt(k), rsk = 1.0 / sk;
    // T: L^{-T} u, MA: L u (MA is dead once S is formed)
    for (int r = NN - 1; r >= 0; --r) {
      double s = V[r * NS + c];
      for (int e = r + 1; e < NN; ++e) s -= LC[e * NS + r] * T[e * NS + c];
      T[r * NS + c] = s / LC[r * NS + r];
    }
    for (int r = NN - 1; r >= 0; --r) {
      double s = 0.0;
      for (int e = 0; e <= r; ++e) s += LC[r * NS + e] * V[e * NS + c];
      MA[r * NS + c] = s;
    }
    for (int r = 0; r < NN; ++r) {
      T[r * NS + c] *= sk;
      MA[r * NS + c] *= rsk;
    }
    const double* x = (primary ? MA : T) + c;
    const double* y = (primary ? T : MA) + c;
    double* vec = q.lrec;
    const double dts = q.rec[q.il.dtau_s + q.lc];
    const double ks = lneg && !primary ? -k : k;  // (the reference's a and b change roles)
    vec[mod_k(N) + c] = ks;
    const double em = expm1(mode_exponent(ks, dts));  // E - 1; 1 - E^2 = -em (2 + em)
    vec[mod_E(N) + c] = 1.0 + em;
    vec[mod_F(N) + c] = -em * (2.0 + em);
    if (beam) {
      double umu0 = q.rec[H_UMU0];
      bool res = false;
      for (int e = 0; e < NN; ++e) res = res || beam_resonant(mode_k(Sc[e * NS + e]), umu0);
      if (res) umu0 = 0.999 * umu0;
      double al = 0.0, be = 0.0;
      for (int r = 0; r < NN; ++r) {
        al += x[r * NS] * b1[r];
        be += y[r * NS] * b2[r];
      }
      const double r0 = 1.0 / umu0, ka = lneg && primary ? -k : k, kb = lneg && !primary ? -k : k;
      const double den = ka * kb - r0 * r0;
      vec[mod_cb(N) + c] = (kb * al - be * r0) / den;
      vec[mod_db(N) + c] = (ka * be - al * r0) / den;
    }
    if (p.flags & DSP_FLAG_THERMAL) {
      double v = 0.0;
      for (int r = 0; r < NN; ++r) v += x[r * NS] * (dsim[r] / mu[r]);
      v = 2.0 * (1.0 - ws) * v / (lneg && primary ? -k : k);
      vec[mod_ct(N) + c] = v;
      vec[mod_dt(N) + c] = v / (lneg && !primary ? -k : k);
      if (c == 0) thermal_source(q, vec[mod_xr(N)], vec[mod_xr(N) + 1]);
    }
  }
  team_sync<TEAM>();
  {
    const double* X = primary ? MA : T;
    const double* Yv = primary ? T : MA;
    for (int it = t; it < NN * HP; it += TEAM) {
      const int c = it / HP, r = it % HP;
      q.lrec[mod_X(N) + it] = r < NN ? X[r * NS + c] : 0.0;
      q.lrec[mod_Y(N) + it] = r < NN ? Yv[r * NS + c] : 0.0;
    }
  }
}

// Pivot of a Cholesky factorisation, d0 the diagonal element it started from: at
// omega' = 1 the last pivot of -A_s is zero to rounding, of either sign, and is
// taken as 1e-18 d0 (k ~ 1e-9); NaN or a negative pivot beyond rounding: 0, the
// matrix is indefinite.
__device__ __forceinline__ double chol_pivot(double s, double d0) {
  return s > 1e-18 * d0 ? s : (s > -1e-12 * d0 ? 1e-18 * d0 : 0.0);
}

// Cholesky of a packed lower triangle in place; false when the matrix is
// indefinite (the factor is then not used).
template <int NN>
__device__ __forceinline__ bool chol_packed(double* A) {
  bool ok = true;
#pragma unroll
  for (int j = 0; j < NN; ++j) {
    const double d0 = A[tri_idx(j, j)];
    double s = d0;
#pragma unroll
    for (int k = 0; k < j; ++k) s -= A[tri_idx(j, k)] * A[tri_idx(j, k)];
    s = chol_pivot(s, d0);
    ok = ok && s > 0.0;
    const double r = rsqrt(ok ? s : 1.0);
    A[tri_idx(j, j)] = ok ? s * r : 1.0;
#pragma unroll
    for (int i = j + 1; i < NN; ++i) {
      double t = A[tri_idx(i, j)];
#pragma unroll
      for (int k = 0; k < j; ++k) t -= A[tri_idx(i, k)] * A[tri_idx(j, k)];
      A[tri_idx(i, j)] = t * r;
    }
  }
  return ok;
}

// An indefinite S is shifted by the first of kFirstShift x its largest row sum, 16 times
// that, ... that makes it positive definite: not far above its most negative eigenvalue,
// so that the small eigenvalues keep their digits, and at the row sum at the latest.
constexpr double kFirstShift = 1.0e-6;

// The front's hand-off of a task with exactly one of -B_s (okb) and -A_s positive
// definite: S = L^T M L with the definite one's factor L and the other as M, shifted
// and scaled for onesided_jacobi.  Rare (phase functions with unphysical moments):
// local memory and rolled loops.
template <int N, bool GEN>
__device__ __noinline__ void layer_front_indefinite(const FluxParams& p, const LayerTask<N, GEN>& q, double* hand,
                                                    long long nt, long long j, bool okb) {
  constexpr int NN = N / 2;
  using HO = Handoff<NN>;
  const int m = mode_of<GEN>(p);
  const double* tab = p.tables + mode_row<GEN>() * (long long)tab_size(N);
  const double* Y = tab + tab_ylm(N);
  double M[2][HO::TRI], gl[N];  // -B_s, -A_s
  const double ws = q.rec[q.il.ssa_s + q.lc], f = q.rec[q.il.fsc + q.lc], sig = q.rec[q.il.sig + q.lc];
  const int mode = (int)q.rec[q.il.mode + q.lc];
  for (int k = 0; k < N; ++k) gl[k] = phase_coeff<GEN>(k, q.pml[k], mode, ws, f, sig);
  for (int r = 0; r < NN; ++r)
    for (int c = 0; c <= r; ++c) {
      double sum[2] = {0.0, 0.0};  // odd, even l + m
      for (int l = 0; l < N; ++l) sum[1 - ((l + m) & 1)] += gl[l] * Y[l * N + r] * Y[l * N + c];
      const double rm = 1.0 / tab[tab_mu(N) + r];
      for (int h = 0; h < 2; ++h)
        M[h][tri_idx(r, c)] = -tab[tab_dsim(N) + r] * ((tab[tab_wt(N) + c] * sum[h]) * rm - (r == c ? rm : 0.0)) *
                              tab[tab_dinv(N) + c];
    }
  double* const L = okb ? M[0] : M[1];
  double* const I = okb ? M[1] : M[0];  // the indefinite one, then scratch
  for (int c = 0; c < NN; ++c) {
    const double d0 = L[tri_idx(c, c)];
    double v = d0;
    for (int k = 0; k < c; ++k) v -= L[tri_idx(c, k)] * L[tri_idx(c, k)];
    const double ljj = sqrt(chol_pivot(v, d0));
    L[tri_idx(c, c)] = ljj;
    for (int r = c + 1; r < NN; ++r) {
      double t = L[tri_idx(r, c)];
      for (int k = 0; k < c; ++k) t -= L[tri_idx(r, k)] * L[tri_idx(c, k)];
      L[tri_idx(r, c)] = t / ljj;
    }
  }
  double S[HO::TRI];
  for (int c = 0; c < NN; ++c) {
    double t[NN];  // (M L)[:, c]
    for (int r = 0; r < NN; ++r) {
      t[r] = 0.0;
      for (int k = c; k < NN; ++k) t[r] += I[tri_idx(r, k)] * L[tri_idx(k, c)];
    }
    for (int r = c; r < NN; ++r) {
      double v = 0.0;
      for (int k = r; k < NN; ++k) v += L[tri_idx(k, r)] * t[k];
      S[tri_idx(r, c)] = v;
    }
  }
  double scale = 0.0;  // largest row sum: no eigenvalue is beyond it
  for (int r = 0; r < NN; ++r) {
    double v = 0.0;
    for (int c = 0; c < NN; ++c) v += fabs(S[tri_idx(r, c)]);
    scale = fmax(scale, v);
  }
  if (!(scale > 0.0)) scale = 1.0;
  double shift = kFirstShift * scale;
  for (; shift < scale; shift *= 16.0) {
    bool ok = true;
    for (int c = 0; c < NN && ok; ++c)
      for (int r = c; r < NN; ++r) {
        double v = S[tri_idx(r, c)] + (r == c ? shift : 0.0);
        for (int k = 0; k < c; ++k) v -= I[tri_idx(r, k)] * I[tri_idx(c, k)];
        if (r == c) ok = v > 0.0;
        I[tri_idx(r, c)] = r == c ? sqrt(fmax(v, 0.0)) : v / I[tri_idx(c, c)];
      }
    if (ok) break;
  }
  for (int c = 0; c < NN; ++c)
    for (int r = 0; r < NN; ++r)
      *handoff_lane<NN>(hand, nt, j, HO::S_F + c * NN + r) = (S[tri_idx(r, c)] + (r == c ? shift : 0.0)) / scale;
  q.lrec[mod_xr(N)] = shift;
  q.lrec[mod_xr(N) + 1] = scale;
  for (int e = 0; e < HO::TRI; ++e) *handoff_lane<NN>(hand, nt, j, HO::S_L + e) = L[e];
  *handoff_lane<NN>(hand, nt, j, HO::S_FLAG) = okb ? 2.0 : 3.0;
}

// ---------------------------------------------------------------------------
// Front of a split layer stage, one thread per layer task: scaled phase
// coefficients (disortSet, FluxSolver.cpp:336-386), the phase sums, alpha -/+ beta
// in the symmetric form of the reference (FluxSolver.cpp:466-514), the Cholesky
// factors of -B_s and -A_s (:521-558), L^T R and the beam's source vectors,
// written to the hand-off.  Every matrix is a packed symmetric
// h x h in registers; the tables are constant-bank operands.
// ---------------------------------------------------------------------------
template <int N, bool GEN>
__global__ void __launch_bounds__(128) flux_layer_front_kernel(FluxParams p, ConstTab<N> tc) {
  constexpr int NN = N / 2;
  using HO = Handoff<NN>;
  constexpr int TRI = HO::TRI;
  // P_l^m(mu_i): the flux path's from the constant bank, the general solver's (one
  // table per mode of the launch) from shared memory, read where it is used
  // (volatile: kept in registers over the sums, the table would push them to
  // local memory)
  __shared__ double ysm[GEN ? N * NN : 1];
  if constexpr (GEN) {
    const double* Y = p.tables + (long long)mode_row<GEN>() * tab_size(N) + tab_ylm(N);
    for (int e = threadIdx.x; e < N * NN; e += blockDim.x) ysm[e] = Y[(e / NN) * N + e % NN];
    __syncthreads();
  }
  const volatile double* const yv = ysm;
  auto ytab = [&](int l, int i) -> double {
    if constexpr (GEN) return yv[l * NN + i];
    else return tc.y[l * NN + i];
  };
  const long long nt = layer_tasks<GEN>(p);
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nt) return;
  const int m = mode_of<GEN>(p);
  double* const hand = p.bvp_rec + mode_row<GEN>() * p.g.ms_bvp;
  auto hp = [&](int e) { return handoff_lane<NN>(hand, nt, j, e); };
  const LayerTask<N, GEN> q = layer_task<N, GEN>(p, j);
  if (!q.live) {
    *hp(HO::S_FLAG) = 0.0;
    return;
  }
  const double ws = q.rec[q.il.ssa_s + q.lc];
  // ---- phase sums of odd (O) and even (E) l + m ----------------------------
  double O[TRI], E[TRI];
  {
    double gl[N];
    const int mode = (int)q.rec[q.il.mode + q.lc];
    const double f = q.rec[q.il.fsc + q.lc], sig = q.rec[q.il.sig + q.lc];
#pragma unroll
    for (int k = 0; k < N; ++k) gl[k] = phase_coeff<GEN>(k, q.pml[k], mode, ws, f, sig);
#pragma unroll
    for (int a = 0; a < NN; ++a) {
      double z[N];
#pragma unroll
      for (int l = 0; l < N; ++l) z[l] = gl[l] * ytab(l, a);
#pragma unroll
      for (int b = 0; b <= a; ++b) {
        double se = 0.0, so = 0.0;
#pragma unroll
        for (int l = 0; l < N; l += 2) se += z[l] * ytab(l, b);
#pragma unroll
        for (int l = 1; l < N; l += 2) so += z[l] * ytab(l, b);
        E[tri_idx(a, b)] = se;
        O[tri_idx(a, b)] = so;
      }
    }
    const double fbeam = q.rec[H_FBEAM];
    const bool swap = GEN && (m & 1);
    if (fbeam > 0.0) {
      // (2 - delta_m0) F0 / 4pi sum_k g'_k P_k^m(mu_r) P_k^m(-mu0) by parity (DisortSolver.cpp:1361-1368)
      const double* yb = beam_legendre<N, GEN>(p, q);
#pragma unroll
      for (int k = 0; k < N; ++k) gl[k] *= yb[k];
      const double fac = ((GEN && m > 0) ? 4.0 : 2.0) * fbeam / (4.0 * 3.14159265358979323846);
#pragma unroll
      for (int r = 0; r < NN; ++r) {
        double se = 0.0, so = 0.0;
#pragma unroll
        for (int l = 0; l < N; l += 2) se += gl[l] * ytab(l, r);
#pragma unroll
        for (int l = 1; l < N; l += 2) so += gl[l] * ytab(l, r);
        const double dm = tc.dsim[r] * tc.rmu[r] * fac;
        *hp(HO::S_B1 + r) = dm * (swap ? so : se);
        *hp(HO::S_B2 + r) = dm * (swap ? se : so);
      }
    }
    if (swap) {
#pragma unroll
      for (int e = 0; e < TRI; ++e) {
        const double x = O[e];
        O[e] = E[e];
        E[e] = x;
      }
    }
  }
  // -B_s = -D (a-b) D^{-1} and -A_s = -D (a+b) D^{-1} (packed lower; both symmetric)
  auto minus_s = [&](const double* P, double* X) {
#pragma unroll
    for (int r = 0; r < NN; ++r)
#pragma unroll
      for (int c = 0; c <= r; ++c) {
        const double a = (tc.wt[c] * P[tri_idx(r, c)]) * tc.rmu[r] - (r == c ? tc.rmu[r] : 0.0);
        X[tri_idx(r, c)] = -tc.dsim[r] * a * tc.dinv[c];
      }
  };
  // ---- Cholesky factors L of -B_s and R of -A_s, F = L^T R -------------------
  double Lf[TRI], R[TRI];
  minus_s(O, Lf);
  minus_s(E, R);
  const bool okb = chol_packed<NN>(Lf), oka = chol_packed<NN>(R);
  if (okb && oka) {
#pragma unroll
    for (int c = 0; c < NN; ++c)
#pragma unroll
      for (int r = 0; r < NN; ++r) {
        double v = 0.0;
#pragma unroll
        for (int k = (r > c ? r : c); k < NN; ++k) v += Lf[tri_idx(k, r)] * R[tri_idx(k, c)];
        *hp(HO::S_F + c * NN + r) = v;
      }
#pragma unroll
    for (int e = 0; e < TRI; ++e) *hp(HO::S_L + e) = Lf[e];
    *hp(HO::S_FLAG) = 1.0;
    return;
  }
  if (!okb && !oka) {
    no_eigensystem<N, GEN>(p, q);
    *hp(HO::S_FLAG) = 0.0;
    return;
  }
  layer_front_indefinite<N, GEN>(p, q, hand, nt, j, okb);
}

// Tangent of the Jacobi angle that makes two columns of squared norms app, aqq and
// inner product apq orthogonal (0 where they are to rounding): the smaller root t
// of t^2 + 2 th t - 1, th = (aqq - app) / (2 apq).  In single precision: the
// rotation built from it is orthogonal to double precision whatever t is
// (rsqrt_near1), and an angle off by 1e-7 of itself leaves 1e-7 of the inner
// product, which the next sweep's quadratic convergence absorbs.
// far: the pair was rotated by more than 1e-8 or was further than 1e-8 from
// orthogonal.
__device__ __forceinline__ float jacobi_tan(double apq, double app, double aqq, bool& far) {
  const double g2 = apq * apq, ab = app * aqq;
  const bool need = g2 > DSP_JACOBI_TOL2 * ab;
  const float d = static_cast<float>(aqq - app), e = 2.0f * static_cast<float>(apq);
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fmaf(d, d, e * e)));
  // columns of equal norm turn by 45 degrees; there the approximations give up to 1 + 2^-23
  const float t = fminf(__fdividef(fabsf(e), fabsf(d) + r), 1.0f);
  const bool use = need && e != 0.0f;
  far = use && (t > 1e-8f || g2 > 1e-16 * ab);
  const bool same = (d < 0.0f) == (e < 0.0f);  // sgn(th), sgn(0) = +1
  return use ? (same ? t : -t) : 0.0f;
}

// 1/sqrt(x) for x in [1, 2]: the single-precision value y refined by one step of
// the third-order iteration y (1 + e/2 + 3 e^2/8), e = 1 - x y^2 (e ~ 2^-22, error
// ~ e^3; Muller et al., Handbook of Floating-Point Arithmetic, section 4.7).
__device__ __forceinline__ double rsqrt_near1(double x) {
  const double y = static_cast<double>(rsqrtf(static_cast<float>(x)));
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// One round of a one-sided Jacobi sweep in odd-even order: the pairs (p, p + 1),
// p = ODD, ODD + 2, ..., of the columns of F are rotated to be orthogonal and change
// places, so that n rounds bring every two columns together, always in the same
// registers.  nrm: the columns' squared norms.  Returns whether a pair was rotated
// by more than 1e-8 or its columns were further than 1e-8 from orthogonal: when
// none of a sweep's was, what is left is below rounding (quadratic convergence,
// and the angles' 1e-7).  live: false leaves the columns in place, up to sign.
template <int NN, int ODD>
__device__ __forceinline__ bool onesided_round(double (*F)[NN], double* nrm, bool live) {
  constexpr int NPAIR = (NN - ODD) / 2;
  bool more = false;
  // the rotations of the round's pairs side by side (their serial chains overlap)
  double cs[NPAIR > 0 ? NPAIR : 1], sn[NPAIR > 0 ? NPAIR : 1];
#pragma unroll
  for (int a = 0; a < NPAIR; ++a) {
    const int p = 2 * a + ODD, q = p + 1;
    double d0 = 0.0, d1 = 0.0;
#pragma unroll
    for (int r = 0; r < NN; r += 2) {
      d0 = fma(F[p][r], F[q][r], d0);
      if (r + 1 < NN) d1 = fma(F[p][r + 1], F[q][r + 1], d1);
    }
    const double g = d0 + d1, np = nrm[p], nq = nrm[q];
    bool far;
    const float tf = jacobi_tan(g, np, nq, far);
    const double t = tf;
    more = more || far;
    const double c = rsqrt_near1(fma(t, t, 1.0));
    cs[a] = live ? c : 0.0;  // a finished task's columns stay in place (one changes sign)
    sn[a] = live ? t * c : 1.0;
    nrm[q] = fma(-t, g, np);
    nrm[p] = fma(t, g, nq);
  }
#pragma unroll
  for (int a = 0; a < NPAIR; ++a) {
    const int p = 2 * a + ODD, q = p + 1;
#pragma unroll
    for (int r = 0; r < NN; ++r) {
      const double x = F[p][r], y = F[q][r];
      F[q][r] = fma(cs[a], x, -(sn[a] * y));
      F[p][r] = fma(sn[a], x, cs[a] * y);
    }
  }
  return more;
}

// One-sided Jacobi iteration on the columns of F, in registers.  Two rounds are the
// body of a rolled loop (a sweep unrolled overflows the instruction cache: 1.8 of
// 5.5 stalled cycles per instruction; the round-robin order, rolled, moves every
// column between registers).  A warp runs until its last active task has
// converged, 3 to 5 sweeps; a task that has is left as it is, so that its result
// does not depend on the others of its warp.
template <int NN>
__device__ __forceinline__ void onesided_jacobi(double (*F)[NN], bool act) {
  bool live = act;
  for (int sweep = 0; sweep < 20; ++sweep) {
    double nrm[NN];
#pragma unroll
    for (int c = 0; c < NN; ++c) {
      nrm[c] = 0.0;
#pragma unroll
      for (int r = 0; r < NN; ++r) nrm[c] = fma(F[c][r], F[c][r], nrm[c]);
    }
    bool more = false;
#pragma unroll 1
    for (int r = 0; r < NN; r += 2) {
      more = onesided_round<NN, 0>(F, nrm, live) || more;
      more = onesided_round<NN, 1>(F, nrm, live) || more;
    }
    live = live && more;
    if (!__any_sync(0xffffffffu, live)) break;
  }
}

// Eigensolver and output of the split layer stage, one thread per layer task: F
// from the hand-off into registers, onesided_jacobi, then mode by mode X and Y
// (from the singular vector and the Cholesky factor), k and the particular
// solutions in the modes.  The layer record is staged per warp in shared memory
// and written with consecutive lanes on consecutive doubles.
template <int N>
struct ECfg {
  static constexpr int HP = mod_hp(N);
  static constexpr int RS = 2 * HP + 1;   // staging row: one mode's X and Y
  static constexpr int VS = 7 * HP + 3;   // staging row: the vectors
  static constexpr int WARP = 32 * (RS + VS);
  static constexpr size_t smem_bytes(int cta) { return sizeof(double) * (size_t)(cta / 32) * WARP; }
};

template <int N, bool GEN>
__global__ void __launch_bounds__(128) flux_eigen_kernel(FluxParams p, ConstTab<N> tc) {
  constexpr int NN = N / 2;
  using HO = Handoff<NN>;
  using C = ECfg<N>;
  constexpr int HP = C::HP, RS = C::RS, VS = C::VS;
  extern __shared__ double smem[];
  const int lane = threadIdx.x & 31;
  double* const stg = smem + (threadIdx.x >> 5) * C::WARP;
  double* const vst = stg + 32 * RS;
  double* const row = stg + lane * RS;
  double* const vrow = vst + lane * VS;
  const long long nt = layer_tasks<GEN>(p);
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long j0 = j - lane;
  if (j0 >= nt) return;  // whole warp past the end (warp-uniform)
  // lanes past the end or skipped by the front compute on a valid task's
  // addresses and write nothing (no early exit: the warp writes rows together)
  const long long jj = j < nt ? j : nt - 1;
  const int m = mode_of<GEN>(p);
  double* const hand = p.bvp_rec + mode_row<GEN>() * p.g.ms_bvp;
  auto hv = [&](int e) { return *handoff_lane<NN>(hand, nt, jj, e); };
  const double flag = hv(HO::S_FLAG);
  const bool act = j < nt && flag != 0.0;  // skipped: cut layer, invalid input, no factorisation
  const unsigned okm = __ballot_sync(0xffffffffu, act);
  if (okm == 0u) return;  // warp-uniform
  double F[NN][NN], kk[NN];
  const bool regular = flag < 1.5;
#pragma unroll
  for (int c = 0; c < NN; ++c)
#pragma unroll
    for (int r = 0; r < NN; ++r) F[c][r] = act ? hv(HO::S_F + c * NN + r) : 0.0;
  onesided_jacobi<NN>(F, act);
#pragma unroll
  for (int c = 0; c < NN; ++c) {
    double n2 = 0.0;
#pragma unroll
    for (int r = 0; r < NN; ++r) n2 = fma(F[c][r], F[c][r], n2);
    const double rs = n2 > 0.0 ? rsqrt(n2) : 0.0;
    kk[c] = fmax(n2 * rs, 1e-9);
#pragma unroll
    for (int r = 0; r < NN; ++r) F[c][r] *= rs;
  }
  const LayerTask<N, GEN> q = layer_task<N, GEN>(p, jj);
  // eigenvalues lambda = k^2 are negative only where -A_s (bit set in nega) or -B_s
  // (negb) is indefinite; k = sqrt|lambda| as in the reference, the inverses of the
  // particular solutions carry the sign, and with -B_s the reference's a and b
  // change roles, which is the mode of -k
  unsigned nega = 0u, negb = 0u;
  if (act && !regular) {
    const double shift = q.lrec[mod_xr(N)], scale = q.lrec[mod_xr(N) + 1];
#pragma unroll
    for (int c = 0; c < NN; ++c) {
      const double lambda = fma(kk[c], scale, -shift);
      kk[c] = mode_k(lambda);
      if (lambda < 0.0) (flag < 2.5 ? nega : negb) |= 1u << c;
    }
  }

  const bool primary = flag < 2.5;
  const double fbeam = act ? q.rec[H_FBEAM] : 0.0;
  const bool beam = fbeam > 0.0;
  const bool raw = GEN && (p.flags & DSP_FLAG_SPHERICAL_BEAM);
  const bool thermal = (p.flags & DSP_FLAG_THERMAL) && m == 0;
  double r0 = 0.0;
  if (beam) {
    double umu0 = q.rec[H_UMU0];
    bool res = false;
#pragma unroll
    for (int c = 0; c < NN; ++c) res = res || beam_resonant(kk[c], umu0);
    if (res) umu0 = 0.999 * umu0;
    r0 = 1.0 / umu0;
  }
  const double ws2 = act ? 2.0 * (1.0 - q.rec[q.il.ssa_s + q.lc]) : 0.0;
  double L[HO::TRI];
#pragma unroll
  for (int e = 0; e < HO::TRI; ++e) L[e] = act ? hv(HO::S_L + e) : 1.0;
  double rdg[NN];
#pragma unroll
  for (int k = 0; k < NN; ++k) rdg[k] = rcp_newton(L[tri_idx(k, k)]);
  const long long ls = GEN ? p.g.lstride : (long long)lrec_stride(N);
  double* const rec0 = p.layer_rec + mode_row<GEN>() * p.g.ms_layer + j0 * ls;
  const double dts = act ? q.rec[q.il.dtau_s + q.lc] : 0.0;
#pragma unroll
  for (int c = 0; c < NN; ++c) {
    const double k = kk[c], rsk = rsqrt(k), sk = k * rsk;
    double x[NN], y[NN];
    // y = L^{-T} u, x = L u
#pragma unroll
    for (int r = 0; r < NN; ++r) y[r] = F[c][r];
#pragma unroll
    for (int e = NN - 1; e >= 0; --e) {
      y[e] *= rdg[e];
#pragma unroll
      for (int r = 0; r < e; ++r) y[r] -= L[tri_idx(e, r)] * y[e];
    }
#pragma unroll
    for (int r = 0; r < NN; ++r) {
      double s = 0.0;
#pragma unroll
      for (int e = 0; e <= r; ++e) s += L[tri_idx(r, e)] * F[c][e];
      x[r] = s;
    }
    double ve = 0.0, al = 0.0, be = 0.0;
#pragma unroll
    for (int r = 0; r < NN; ++r) {
      const double lu = x[r] * rsk, li = y[r] * sk;
      x[r] = primary ? lu : li;
      y[r] = primary ? li : lu;
      row[r] = x[r];
      row[HP + r] = y[r];
      ve += x[r] * (tc.dsim[r] * tc.rmu[r]);
    }
    if (HP != NN) {
      row[NN] = 0.0;
      row[HP + NN] = 0.0;
    }
    const double ks = (negb >> c) & 1u ? -k : k;
    vrow[c] = ks;
    const double em = expm1(mode_exponent(ks, dts));  // E - 1; 1 - E^2 = -em (2 + em)
    vrow[HP + c] = 1.0 + em;
    vrow[2 * HP + c] = -em * (2.0 + em);
    if (beam) {
      if (raw) {
        // pseudo-spherical beam (general solver): the raw source at the quadrature
        // angles, up and down, for the user-angle interpolation and
        // flux_sph_source_kernel (DisortSolver.cpp:1524-1527)
        const double dm = 0.5 * tc.mu[c] * tc.dinv[c], u1 = hv(HO::S_B1 + c), u2 = hv(HO::S_B2 + c);
        vrow[3 * HP + c] = dm * (u1 + u2);
        vrow[4 * HP + c] = dm * (u1 - u2);
      } else {
#pragma unroll
        for (int r = 0; r < NN; ++r) {
          al += x[r] * hv(HO::S_B1 + r);
          be += y[r] * hv(HO::S_B2 + r);
        }
        const double ka = (nega >> c) & 1u ? -k : k, kb = (negb >> c) & 1u ? -k : k;
        const double den = rcp_newton(ka * kb - r0 * r0);
        vrow[3 * HP + c] = (kb * al - be * r0) * den;
        vrow[4 * HP + c] = (ka * be - al * r0) * den;
      }
    }
    if (thermal) {
      const double rk = rsk * rsk;
      ve = ws2 * ve * ((nega >> c) & 1u ? -rk : rk);
      vrow[5 * HP + c] = ve;
      vrow[6 * HP + c] = ve * ((negb >> c) & 1u ? -rk : rk);
    }
    // X^T row c and Y^T row c of every task: lane group (task, X or Y) x HP
    __syncwarp();
    constexpr int TPI = 32 / (2 * HP) < 1 ? 1 : 32 / (2 * HP);  // tasks per store
    const int tl = lane / (2 * HP), e = lane % (2 * HP);
    if (tl < TPI)
#pragma unroll 4
      for (int b = tl; b < 32; b += TPI)
        if ((okm >> b) & 1u)
          rec0[b * ls + (e < HP ? mod_X(N) + c * HP + e : mod_Y(N) + c * HP + e - HP)] = stg[b * RS + e];
    __syncwarp();
  }
  if (thermal && act) thermal_source(q, vrow[7 * HP], vrow[7 * HP + 1]);
  __syncwarp();
  for (int b = 0; b < 32; ++b)
    if ((okm >> b) & 1u)
      for (int e = lane; e < 7 * HP + 2; e += 32) rec0[b * ls + mod_k(N) + e] = vst[b * VS + e];
}

// ---------------------------------------------------------------------------
// Layer stage of 32 and 64 streams: a team of h/2 lanes per layer task, two
// columns of h rows per lane in registers (two tasks per warp at 64 streams, four
// at 32).  The same steps as the one-thread stage: phase sums column by column,
// Cholesky factors of -B_s and -A_s with the pivot column exchanged through shared
// memory, F = L^T R, one-sided Jacobi in odd-even order, where a lane's two columns
// are the even rounds' pair and the odd rounds' pair takes the next lane's first
// column by shuffles, and the modes from the triangular factor.
// What bounds it: FP64 issue in the Jacobi rounds (about 5 h + 20 instructions per
// lane and round for two tasks a warp).  The team form it replaced (shared-memory
// two-sided Jacobi with a barrier per round, 128 threads a task at 64 streams) took
// 8.7 ms for 192 x 91 layers at 64 streams, this takes 2.8.
// ---------------------------------------------------------------------------
template <int N>
struct WCfg {
  static constexpr int H = N / 2, TEAM = H / 2, TPW = 32 / TEAM;
  static constexpr int LDM = H + 2;            // row stride: an odd number of 16-byte words
  static constexpr int MAT = H * LDM;
  static constexpr int O_L = 0;                // Cholesky factor L, row-major
  static constexpr int O_R = O_L + MAT;        // -A_s and its factor; then X^T, Y^T on their way out
  static constexpr int O_C = O_R + MAT;        // pivot column, twice (rotated reads), two buffers
  static constexpr int O_GL = O_C + 2 * (2 * H + 4);  // g'_l [N]
  static constexpr int O_B1 = O_GL + N;        // D M^{-1} (q+ + q-), D M^{-1} (q+ - q-), D M^{-1} 1
  static constexpr int O_B2 = O_B1 + H;
  static constexpr int O_E = O_B2 + H;
  static constexpr int SIZE = O_E + H;
  static constexpr int STRIDE = SIZE + ((2 - SIZE) % 16 + 16) % 16;  // teams 4 banks apart
  static constexpr size_t smem_bytes() { return sizeof(double) * (size_t)(TPW * STRIDE); }
  static constexpr int MINB = H == 32 ? 6 : 10;
};

// Cholesky factor of the symmetric matrix whose columns 2t, 2t + 1 lane t holds in
// c0, c1 (rows in order), written row-major to `out` (stride LDM, upper part zero).
// Right-looking; in step k register i of a column is row k + i, the update shifting
// it by one row.  d00, d01: the diagonal elements of the lane's columns (picked out of
// the registers by lane they would put a column into local memory).  Returns false (to
// every lane of the team) if it is indefinite.  STORE = false: only the verdict.
template <int H, int LDM, int TEAM, bool STORE = true>
__device__ __forceinline__ bool team_chol_columns(double* c0, double* c1, double d00, double d01, double* out,
                                                  double* cbuf, int t, unsigned msk) {
  bool ok = true;
#pragma unroll 1
  for (int k2 = 0; k2 < H; k2 += 2) {
#pragma unroll
    for (int odd = 0; odd < 2; ++odd) {
      const int k = k2 + odd;
      const bool mine = t == k2 / 2;
      double* const buf = cbuf + odd * (2 * H + 4);
      if (mine) {
        // register 0 is the pivot
        const double* c = odd ? c1 : c0;
        const double s = chol_pivot(c[0], odd ? d01 : d00);
        const double r = s > 0.0 ? rsqrt(s) : 0.0;
#pragma unroll
        for (int i = 0; i < H; ++i) {
          const double v = i == 0 ? s * r : c[i] * r;
          buf[i] = v;  // rows k .. k + H - 1: past the matrix the registers hold zeros
          if (STORE && k + i < H) out[(k + i) * LDM + k] = v;
        }
        if constexpr (STORE)
          for (int i = 0; i < k; ++i) out[i * LDM + k] = 0.0;
      }
      __syncwarp(msk);
      ok = ok && buf[0] > 0.0;
      // rows of the lane's columns in this step's numbering: column c is row c - k
      const int a0 = 2 * t - k, a1 = a0 + 1;
      const double l0 = a0 > 0 ? buf[a0] : 0.0, l1 = a1 > 0 ? buf[a1] : 0.0;
      const double2* b2 = reinterpret_cast<const double2*>(buf);
      {
        const double2 w = b2[0];
        c0[0] = fma(-l0, w.y, c0[1]);
        c1[0] = fma(-l1, w.y, c1[1]);
      }
#pragma unroll
      for (int i = 2; i < H; i += 2) {
        const double2 w = b2[i / 2];
        c0[i - 1] = fma(-l0, w.x, c0[i]);
        c1[i - 1] = fma(-l1, w.x, c1[i]);
        c0[i] = fma(-l0, w.y, c0[i + 1]);
        c1[i] = fma(-l1, w.y, c1[i + 1]);
      }
      c0[H - 1] = 0.0;
      c1[H - 1] = 0.0;
    }
  }
  __syncwarp(msk);
  return ok;
}

// One-sided Jacobi iteration on a team's columns (two per lane) in odd-even order: a
// lane's two columns are the even rounds' pair, the odd rounds' pair takes the next
// lane's first column by shuffles.  Leaves the columns normalised and their norms in k0,
// k1.  live: false leaves the columns in place, up to sign.  The warp goes together.
template <int H, int TEAM>
__device__ __forceinline__ void team_onesided_jacobi(double* F0, double* F1, double& k0, double& k1, bool live, int t) {
  const unsigned msk = 0xffffffffu;
  auto dot = [](const double* x, const double* y) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
    for (int r = 0; r < H; r += 4) {
      s0 = fma(x[r], y[r], s0);
      s1 = fma(x[r + 1], y[r + 1], s1);
      s2 = fma(x[r + 2], y[r + 2], s2);
      s3 = fma(x[r + 3], y[r + 3], s3);
    }
    return (s0 + s1) + (s2 + s3);
  };
  const bool last = t == TEAM - 1;
#pragma unroll 1
  for (int sweep = 0; sweep < 20; ++sweep) {
    double n0 = dot(F0, F0), n1 = dot(F1, F1);
    bool more = false;
#pragma unroll 1
    for (int rd = 0; rd < H; rd += 2) {
      {  // even round: the lane's own pair, changing places
        bool far;
        const double g = dot(F0, F1);
        const double tn = jacobi_tan(g, n0, n1, far);
        more = more || far;
        const double cc = rsqrt_near1(fma(tn, tn, 1.0));
        const double c = live ? cc : 0.0, s = live ? tn * cc : 1.0;
        const double q0 = n0, q1 = n1;
        n1 = live ? fma(-tn, g, q0) : q1;
        n0 = live ? fma(tn, g, q1) : q0;
#pragma unroll
        for (int r = 0; r < H; ++r) {
          const double x = F0[r], y = F1[r];
          F1[r] = fma(c, x, -(s * y));
          F0[r] = fma(s, x, c * y);
        }
      }
      {  // odd round: the second column with the next lane's first, changing places
        double G[H];
#pragma unroll
        for (int r = 0; r < H; ++r) G[r] = __shfl_down_sync(msk, F0[r], 1, TEAM);
        const double ng = __shfl_down_sync(msk, n0, 1, TEAM);
        bool far;
        const double g = dot(F1, G);
        const double tn = jacobi_tan(g, n1, ng, far);
        const bool rot = live && !last;
        more = more || (far && !last);
        const double cc = rsqrt_near1(fma(tn, tn, 1.0));
        const double c = rot ? cc : 0.0, s = rot ? tn * cc : 1.0;
        const double qn = rot ? fma(-tn, g, n1) : ng;  // squared norm of the column handed on
        n1 = rot ? fma(tn, g, ng) : n1;
#pragma unroll
        for (int r = 0; r < H; ++r) {
          const double x = F1[r], y = G[r];
          G[r] = fma(c, x, -(s * y));
          F1[r] = fma(s, x, c * y);
          const double back = __shfl_up_sync(msk, G[r], 1, TEAM);
          F0[r] = t == 0 ? F0[r] : back;
        }
        const double nb = __shfl_up_sync(msk, qn, 1, TEAM);
        n0 = t == 0 ? n0 : nb;
      }
    }
    // the task's verdict is the team's
    const unsigned tm = __ballot_sync(msk, live && more);
    const unsigned team_bits = (TEAM == 32 ? 0xffffffffu : ((1u << TEAM) - 1u)) << (threadIdx.x & 31u & ~(unsigned)(TEAM - 1));
    live = live && (tm & team_bits) != 0u;
    if (!__any_sync(msk, live)) break;
  }
  k0 = dot(F0, F0);
  k1 = dot(F1, F1);
  {
    const double r0 = k0 > 0.0 ? rsqrt(k0) : 0.0, r1 = k1 > 0.0 ? rsqrt(k1) : 0.0;
    k0 = fmax(k0 * r0, 1e-9);
    k1 = fmax(k1 * r1, 1e-9);
#pragma unroll
    for (int r = 0; r < H; ++r) {
      F0[r] *= r0;
      F1[r] *= r1;
    }
  }
}

// Columns 2t, 2t + 1 of -A_s or -B_s, the phase sums over l = l0, l0 + 2, ..., and their
// diagonal elements once more.
template <int N>
__device__ __forceinline__ void team_matrix_columns(double* F0, double* F1, double& d00, double& d01, int l0, const double* gl, const double* ev,
                                                    const double* Y, const double* tab, int t) {
  constexpr int H = N / 2;
  const double w0 = tab[tab_wt(N) + 2 * t], w1 = tab[tab_wt(N) + 2 * t + 1];
  const double i0 = tab[tab_dinv(N) + 2 * t], i1 = tab[tab_dinv(N) + 2 * t + 1];
  d00 = d01 = 0.0;
#pragma unroll
  for (int r = 0; r < H; ++r) F0[r] = F1[r] = 0.0;
#pragma unroll 1
  for (int l = l0; l < N; l += 2) {
    const double* y = Y + l * N;
    const double z0 = gl[l] * y[2 * t], z1 = gl[l] * y[2 * t + 1];
    d00 = fma(y[2 * t], z0, d00);
    d01 = fma(y[2 * t + 1], z1, d01);
    const double2* y2 = reinterpret_cast<const double2*>(y);
#pragma unroll
    for (int r = 0; r < H; r += 2) {
      const double2 v = y2[r / 2];
      F0[r] = fma(v.x, z0, F0[r]);
      F0[r + 1] = fma(v.y, z0, F0[r + 1]);
      F1[r] = fma(v.x, z1, F1[r]);
      F1[r + 1] = fma(v.y, z1, F1[r + 1]);
    }
  }
#pragma unroll
  for (int r = 0; r < H; ++r) {
    const double dm = ev[r];  // d_r / mu_r
    F0[r] = -dm * (w0 * F0[r] - (r == 2 * t ? 1.0 : 0.0)) * i0;
    F1[r] = -dm * (w1 * F1[r] - (r == 2 * t + 1 ? 1.0 : 0.0)) * i1;
  }
  d00 = -ev[2 * t] * (w0 * d00 - 1.0) * i0;
  d01 = -ev[2 * t + 1] * (w1 * d01 - 1.0) * i1;
}

// Columns 2t, 2t + 1 of A^T C, both in shared memory by rows.
template <int H, int LDM>
__device__ __forceinline__ void team_row_products(double* F0, double* F1, const double* A, const double* C, int t) {
#pragma unroll
  for (int r = 0; r < H; ++r) F0[r] = F1[r] = 0.0;
#pragma unroll 1
  for (int k = 0; k < H; ++k) {
    const double c0 = C[k * LDM + 2 * t], c1 = C[k * LDM + 2 * t + 1];
    const double2* a2 = reinterpret_cast<const double2*>(A + k * LDM);
#pragma unroll
    for (int r = 0; r < H; r += 2) {
      const double2 v = a2[r / 2];
      F0[r] = fma(v.x, c0, F0[r]);
      F0[r + 1] = fma(v.y, c0, F0[r + 1]);
      F1[r] = fma(v.x, c1, F1[r]);
      F1[r + 1] = fma(v.y, c1, F1[r + 1]);
    }
  }
}

// INDEF: the pass over the tasks of which exactly one of -B_s and -A_s is positive
// definite (rare: unphysical moments).  The ordinary pass marks them in their
// boundary-value records (dead until the boundary-value kernel) and writes nothing more;
// this one takes the definite matrix's factor L, forms S = L^T M L of the other one, M,
// and goes on from S shifted and scaled as in layer_front_indefinite.  A pass of its own
// costs a launch that finds nothing marked (2 us); as a branch the rare path took registers
// from the ordinary one (192 x 91 layers at 64 streams 2.85 -> 3.85 ms), and one lane per
// task with a two-sided Jacobi in global memory took 110 ms for 192 x 16 marked layers.
template <int N, bool GEN, bool INDEF = false>
__global__ void __launch_bounds__(32, WCfg<N>::MINB) flux_layer_warp_kernel(FluxParams p) {
  using C = WCfg<N>;
  constexpr int H = C::H, TEAM = C::TEAM, LDM = C::LDM;
  extern __shared__ double smem[];
  const int t = threadIdx.x % TEAM;
  const unsigned msk = 0xffffffffu;  // the warp's teams go together
  double* const sm = smem + (threadIdx.x / TEAM) * C::STRIDE;
  double* const Ls = sm + C::O_L;
  double* const Rs = sm + C::O_R;
  double* const cb = sm + C::O_C;
  double* const gl = sm + C::O_GL;
  double* const b1 = sm + C::O_B1;
  double* const b2 = sm + C::O_B2;
  double* const ev = sm + C::O_E;
  const int m = mode_of<GEN>(p);
  const double* const tab = p.tables;
  const double* const Y = tab + (long long)mode_row<GEN>() * tab_size(N) + tab_ylm(N);
  const long long nt = layer_tasks<GEN>(p);
  const long long task = (long long)blockIdx.x * C::TPW + threadIdx.x / TEAM;
  // a team without a task computes on the last one's inputs and writes nothing
  double* const mark = p.bvp_rec + mode_row<GEN>() * p.g.ms_bvp + task * brec_stride(N);
  const bool marked = INDEF && task < nt && *mark != 0.0;  // (of layers not solved: anything)
  if (INDEF && !__any_sync(msk, marked)) return;
  const LayerTask<N, GEN> q = layer_task<N, GEN>(p, task < nt ? task : nt - 1);
  bool act = task < nt && q.live && (!INDEF || marked);
  if (!__any_sync(msk, act)) return;
  const double ws = q.rec[q.il.ssa_s + q.lc];
  {
    const int mode = (int)q.rec[q.il.mode + q.lc];
    const double f = q.rec[q.il.fsc + q.lc], sig = q.rec[q.il.sig + q.lc];
    for (int k = t; k < N; k += TEAM) gl[k] = phase_coeff<GEN>(k, q.pml[k], mode, ws, f, sig);
  }
  __syncwarp(msk);
  const int odd0 = 1 - (m & 1);  // first l of odd l + m
  const double fbeam = act ? q.rec[H_FBEAM] : 0.0;
  const bool beam = fbeam > 0.0;
  for (int r = t; r < H; r += TEAM) {
    const double dm = tab[tab_dsim(N) + r] / tab[r];
    ev[r] = dm;
    double so = 0.0, se = 0.0;
    if (beam) {
      // (2 - delta_m0) F0 / 4pi sum_k g'_k P_k^m(mu_r) P_k^m(-mu0) by parity (DisortSolver.cpp:1361-1368)
      const double* yb = beam_legendre<N, GEN>(p, q);
      const double fac = ((GEN && m > 0) ? 4.0 : 2.0) * fbeam / (4.0 * 3.14159265358979323846);
      for (int l = 0; l < N; l += 2) {
        so += gl[l + odd0] * Y[(l + odd0) * N + r] * yb[l + odd0];
        se += gl[l + 1 - odd0] * Y[(l + 1 - odd0) * N + r] * yb[l + 1 - odd0];
      }
      so *= dm * fac;
      se *= dm * fac;
    }
    b1[r] = se;
    b2[r] = so;
  }
  // ---- columns 2t, 2t + 1 of -A_s (into R) and -B_s (into L) -----------------
  bool ok[2];
  double F0[H], F1[H];
#pragma unroll 1
  for (int part = 0; part < 2; ++part) {  // 0: -A_s (even sums), 1: -B_s (odd sums)
    double d00, d01;
    team_matrix_columns<N>(F0, F1, d00, d01, part == 0 ? 1 - odd0 : odd0, gl, ev, Y, tab, t);
    ok[part] = team_chol_columns<H, LDM, TEAM>(F0, F1, d00, d01, part == 0 ? Rs : Ls, cb, t, msk);
  }
  const bool okb = ok[1], oka = ok[0];
  // lambda = k^2 negative: -A_s (na) or -B_s (nb) indefinite; see flux_eigen_kernel
  bool na0 = false, na1 = false, nb0 = false, nb1 = false;
  double k0, k1;
  if constexpr (!INDEF) {
    if (act && t == 0) {
      *mark = okb != oka ? 1.0 : 0.0;
      if (!okb && !oka) no_eigensystem<N, GEN>(p, q);
    }
    act = act && okb && oka;
    // ---- F = L^T R, columns 2t, 2t + 1 ----------------------------------------
    team_row_products<H, LDM>(F0, F1, Ls, Rs, t);
    team_onesided_jacobi<H, TEAM>(F0, F1, k0, k1, act, t);
  } else {
    auto to_rows = [&] {  // the lane's columns as rows 2t, 2t + 1 of Rs
      __syncwarp(msk);
#pragma unroll
      for (int r = 0; r < H; ++r) {
        Rs[(2 * t) * LDM + r] = F0[r];
        Rs[(2 * t + 1) * LDM + r] = F1[r];
      }
      __syncwarp(msk);
    };
    if (!okb)
      for (int e = t; e < H * H; e += TEAM) Ls[(e / H) * LDM + e % H] = Rs[(e / H) * LDM + e % H];
    double d00, d01;
    team_matrix_columns<N>(F0, F1, d00, d01, okb ? 1 - odd0 : odd0, gl, ev, Y, tab, t);
    to_rows();
    team_row_products<H, LDM>(F0, F1, Rs, Ls, t);  // M L (M is symmetric)
    __syncwarp(msk);
#pragma unroll
    for (int r = 0; r < H; ++r) {
      Rs[r * LDM + 2 * t] = F0[r];
      Rs[r * LDM + 2 * t + 1] = F1[r];
    }
    __syncwarp(msk);
    team_row_products<H, LDM>(F0, F1, Ls, Rs, t);  // S
    to_rows();
    double scale = 0.0, s1 = 0.0;
#pragma unroll
    for (int r = 0; r < H; ++r) {
      scale += fabs(F0[r]);
      s1 += fabs(F1[r]);
    }
    scale = fmax(scale, s1);
#pragma unroll
    for (int off = TEAM / 2; off > 0; off >>= 1) scale = fmax(scale, __shfl_xor_sync(msk, scale, off, TEAM));
    if (!(scale > 0.0)) scale = 1.0;
    double shift = kFirstShift * scale;
    auto shifted = [&] {
#pragma unroll
      for (int r = 0; r < H; ++r) {
        F0[r] = Rs[(2 * t) * LDM + r] + (r == 2 * t ? shift : 0.0);
        F1[r] = Rs[(2 * t + 1) * LDM + r] + (r == 2 * t + 1 ? shift : 0.0);
      }
    };
    bool done = !act;
#pragma unroll 1
    while (!__all_sync(msk, done)) {
      shifted();
      const bool pd = team_chol_columns<H, LDM, TEAM, false>(F0, F1, Rs[(2 * t) * LDM + 2 * t] + shift,
                                                             Rs[(2 * t + 1) * LDM + 2 * t + 1] + shift, nullptr, cb, t, msk);
      if (!done && !pd) shift *= 16.0;
      done = done || pd || !(shift < scale);
    }
    shifted();
#pragma unroll
    for (int r = 0; r < H; ++r) {
      F0[r] /= scale;
      F1[r] /= scale;
    }
    __syncwarp(msk);
    team_onesided_jacobi<H, TEAM>(F0, F1, k0, k1, act, t);
    const double d0 = fma(k0, scale, -shift), d1 = fma(k1, scale, -shift);
    k0 = mode_k(d0);
    k1 = mode_k(d1);
    na0 = okb && d0 < 0.0;
    na1 = okb && d1 < 0.0;
    nb0 = !okb && d0 < 0.0;
    nb1 = !okb && d1 < 0.0;
  }
  const bool primary = !INDEF || okb;  // L factors -B_s
  // ---- x = L u / sqrt(k) (primary; else sqrt(k) L u / k) and its sums ----------
  const double rs0 = rsqrt(k0), rs1 = rsqrt(k1), sk0 = k0 * rs0, sk1 = k1 * rs1;
  // sums of the form with L u (lu) and with L^{-T} u (li): with b1, b2 and D M^{-1} 1
  double lu_b[2] = {0.0, 0.0}, li_b[2] = {0.0, 0.0}, lu_e[2] = {0.0, 0.0}, li_e[2] = {0.0, 0.0};
  const double* const blu = primary ? b1 : b2;  // X goes with b1, Y with b2
  const double* const bli = primary ? b2 : b1;
  double* const outlu = q.lrec + (primary ? mod_X(N) : mod_Y(N));
  double* const outli = q.lrec + (primary ? mod_Y(N) : mod_X(N));
#pragma unroll 1
  for (int r = 0; r < H; ++r) {
    const double2* l2 = reinterpret_cast<const double2*>(Ls + r * LDM);
    double a0 = 0.0, a1 = 0.0, c0 = 0.0, c1 = 0.0;
#pragma unroll
    for (int e = 0; e < H; e += 2) {
      const double2 v = l2[e / 2];
      a0 = fma(v.x, F0[e], a0);
      c0 = fma(v.y, F0[e + 1], c0);
      a1 = fma(v.x, F1[e], a1);
      c1 = fma(v.y, F1[e + 1], c1);
    }
    const double x0 = (a0 + c0) * rs0, x1 = (a1 + c1) * rs1;
    Rs[(2 * t) * LDM + r] = x0;
    Rs[(2 * t + 1) * LDM + r] = x1;
    lu_b[0] = fma(x0, blu[r], lu_b[0]);
    lu_b[1] = fma(x1, blu[r], lu_b[1]);
    lu_e[0] = fma(x0, ev[r], lu_e[0]);
    lu_e[1] = fma(x1, ev[r], lu_e[1]);
  }
  __syncwarp(msk);
  if (act)
    for (int e = t; e < H * H / 2; e += TEAM) {
      const int c = e / (H / 2), r = 2 * (e % (H / 2));
      *reinterpret_cast<double2*>(outlu + c * H + r) = *reinterpret_cast<const double2*>(Rs + c * LDM + r);
    }
  __syncwarp(msk);
  // ---- L^{-T} u sqrt(k): back substitution, fully unrolled ----------------------
#pragma unroll
  for (int e = H - 1; e >= 0; --e) {
    const double2* l2 = reinterpret_cast<const double2*>(Ls + e * LDM);
    const double rd = rcp_newton(Ls[e * LDM + e]);
    const double y0 = F0[e] * rd, y1 = F1[e] * rd;
#pragma unroll
    for (int r = 0; r < e; r += 2) {
      const double2 v = l2[r / 2];
      F0[r] = fma(-v.x, y0, F0[r]);
      F1[r] = fma(-v.x, y1, F1[r]);
      if (r + 1 < e) {
        F0[r + 1] = fma(-v.y, y0, F0[r + 1]);
        F1[r + 1] = fma(-v.y, y1, F1[r + 1]);
      }
    }
    const double z0 = y0 * sk0, z1 = y1 * sk1;
    Rs[(2 * t) * LDM + e] = z0;
    Rs[(2 * t + 1) * LDM + e] = z1;
    li_b[0] = fma(z0, bli[e], li_b[0]);
    li_b[1] = fma(z1, bli[e], li_b[1]);
    li_e[0] = fma(z0, ev[e], li_e[0]);
    li_e[1] = fma(z1, ev[e], li_e[1]);
  }
  __syncwarp(msk);
  if (!act) return;
  for (int e = t; e < H * H / 2; e += TEAM) {
    const int c = e / (H / 2), r = 2 * (e % (H / 2));
    *reinterpret_cast<double2*>(outli + c * H + r) = *reinterpret_cast<const double2*>(Rs + c * LDM + r);
  }
  // ---- k, E, F and the particular solutions --------------------------------------
  double umu0 = q.rec[H_UMU0];
  if (beam) {
    const bool res = beam_resonant(k0, umu0) || beam_resonant(k1, umu0);
    const unsigned tmask = team_mask<TEAM>();
    if (__any_sync(tmask, res)) umu0 = 0.999 * umu0;
  }
  const double dts = q.rec[q.il.dtau_s + q.lc], r0 = beam ? 1.0 / umu0 : 0.0;
  const bool thermal = (p.flags & DSP_FLAG_THERMAL) && m == 0;
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    const int c = 2 * t + v;
    const double k = v ? k1 : k0;
    const bool na = v ? na1 : na0, nb = v ? nb1 : nb0;
    const double ka = na ? -k : k, kb = nb ? -k : k;
    const double em = expm1(mode_exponent(kb, dts));  // E - 1; 1 - E^2 = -em (2 + em)
    q.lrec[mod_k(N) + c] = kb;
    q.lrec[mod_E(N) + c] = 1.0 + em;
    q.lrec[mod_F(N) + c] = -em * (2.0 + em);
    if (beam) {
      if (GEN && (p.flags & DSP_FLAG_SPHERICAL_BEAM)) {
        // pseudo-spherical beam: the raw source at the quadrature angles (DisortSolver.cpp:1524-1527)
        const double dm = 0.5 / ev[c];
        q.lrec[mod_cb(N) + c] = dm * (b1[c] + b2[c]);
        q.lrec[mod_db(N) + c] = dm * (b1[c] - b2[c]);
      } else {
        const double al = primary ? lu_b[v] : li_b[v], be = primary ? li_b[v] : lu_b[v];
        const double den = ka * kb - r0 * r0;
        q.lrec[mod_cb(N) + c] = (kb * al - be * r0) / den;
        q.lrec[mod_db(N) + c] = (ka * be - al * r0) / den;
      }
    }
    if (thermal) {
      const double ct = 2.0 * (1.0 - ws) * (primary ? lu_e[v] : li_e[v]) / ka;
      q.lrec[mod_ct(N) + c] = ct;
      q.lrec[mod_dt(N) + c] = ct / kb;
    }
  }
  if (thermal && t == 0) thermal_source(q, q.lrec[mod_xr(N)], q.lrec[mod_xr(N) + 1]);
}

// Host side of the layer stage, launched through `wrap(kind, launch)`, which may time
// it (kind 0: front, 1: eigensolver, 2: one kernel, or either pass of the warp kernel);
// `host_tab` is a host copy of the (mode's) tab_* tables of N.
template <int N, bool GEN = false>
inline void flux_layer_set_attrs() {
  if constexpr (layer_split<N>()) {
    static_assert(Handoff<N / 2>::HS <= brec_stride(N), "the hand-off must fit in the boundary-value records");
    cudaFuncSetAttribute(flux_eigen_kernel<N, GEN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)ECfg<N>::smem_bytes(128));
  }
  // the team kernel: N <= 16 on the flux path, when a schedule asks for it
  if constexpr (!GEN && layer_split<N>())
    cudaFuncSetAttribute(flux_layer_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LCfg<N>::smem_bytes());
  if constexpr (!layer_split<N>()) {
    cudaFuncSetAttribute(flux_layer_warp_kernel<N, GEN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)WCfg<N>::smem_bytes());
    cudaFuncSetAttribute(flux_layer_warp_kernel<N, GEN, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)WCfg<N>::smem_bytes());
  }
}

// The layer stage of `tasks` layer tasks (of each of `modes` azimuth modes).  N >= 32:
// the warp kernel, twice (INDEF).  N <= 16: front and eigensolver, one thread per task, with `cta`
// threads per CTA (64 or 128), or, when a schedule of the flux path asks for it, the
// team kernel.
template <int N, bool GEN = false, class Wrap>
inline void flux_layer_launch(const FluxParams& p, long long tasks, const double* host_tab, cudaStream_t s,
                              Wrap&& wrap, bool split = layer_split<N>(), int cta = 128, int modes = 1) {
  if constexpr (layer_split<N>()) {
    if (split || GEN) {
      const int b = cta == 64 ? 64 : 128;
      const ConstTab<N> tc = make_const_tab<N>(host_tab);
      const dim3 g((unsigned)((tasks + b - 1) / b), (unsigned)modes);
      wrap(0, [&] { flux_layer_front_kernel<N, GEN><<<g, b, 0, s>>>(p, tc); });
      wrap(1, [&] { flux_eigen_kernel<N, GEN><<<g, b, ECfg<N>::smem_bytes(b), s>>>(p, tc); });
      return;
    }
    if constexpr (!GEN) {
      using C = LCfg<N>;
      const unsigned grid = (unsigned)((tasks + C::TPC - 1) / C::TPC);
      wrap(2, [&] { flux_layer_kernel<N><<<grid, C::CTA, C::smem_bytes(), s>>>(p); });
    }
  } else {
    using C = WCfg<N>;
    const dim3 grid((unsigned)((tasks + C::TPW - 1) / C::TPW), (unsigned)modes);
    wrap(2, [&] { flux_layer_warp_kernel<N, GEN><<<grid, 32, C::smem_bytes(), s>>>(p); });
    wrap(2, [&] { flux_layer_warp_kernel<N, GEN, true><<<grid, 32, C::smem_bytes(), s>>>(p); });
  }
}

}  // namespace dsp
