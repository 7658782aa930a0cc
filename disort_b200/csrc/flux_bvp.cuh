// flux_bvp.cuh — boundary-value problem and fluxes of one instance, all stream
// counts, on a team of pow2ceil(N/2) lanes of one warp.
//
// Replaces setMatrix (FluxSolver.cpp:838-959), solve0 (:966-1131) and
// computeFluxes (:1138-1287), and their DisortSolver counterparts
// (DisortSolver.cpp:1153-1317, 1669-1920, 1980-2124): the same linear system
// (continuity at every interface, the two boundary conditions), solved without
// forming it.
//
// With h = N/2, D = diag(sqrt(w mu)), phi = D (up + down), psi = D (up - down),
// a layer's modes are phi = X C, psi = Y D_ with X^T Y = I (layer stage) and
//   C = E1 a + E2 b + c_p,   D_ = E2 b - E1 a + d_p,
// E1 = exp(-k (tau - tau_top)), E2 = exp(-k (tau_bot - tau)), c_p and d_p the
// particular solution.  The layers above a depth reflect: psi = A phi + g with a
// symmetric A (reciprocity), A = I, g = -2 D (incoming) at the top.  Through a
// layer, with E = exp(-k dtau):
//   M  = X^T A X,  H = (I + M)^{-1},  Z = (1 - E^2) + 2 E H E,  G = Z^{-1},
//   A' = Y (2 G - I) Y^T,
//   r  = c_t + H (X^T g - d_t - c_t),  q = E r,
//   g' = Y (c_b + d_b + 2 G (q - c_b))            (c, d: particular at top, bottom)
// and back up, from phi at the bottom of the layer:
//   b = G (Y^T phi_b - c_b + q),  c = 2 H E b - r,  a = c - E b,
//   phi_t = X (c + c_t).
// I + M and Z are symmetric positive definite whatever the layer (M is a
// congruence of A, and Z < 2), so both are inverted without pivoting, and no
// growing exponential is formed.  (Unphysical moments above 1 can break that; the
// sweeps then run on an indefinite matrix, scaled by the absolute diagonal, whose signs
// stay; and a mode of -k has a growing E, which leaves G as 1/E^2.)  Two h x h inverses
// and four h^3 products per layer take the place of the N-column elimination of a 3h-row
// panel, about a tenth of its operations; near omega' = 1 (k -> 0) nothing cancels,
// because 1 - E^2 comes from expm1.
//
// Fluxes alone need less on the way up (LEAN, up to 16 streams).  Substituted into
// one another, the three equations are
//   phi_t = W phi_b + f,  W = 2 V G Y^T,  V = X H E,  f = X (c_t - r) + 2 V G (q - c_b),
// and the fluxes of a level are sums w (phi +- psi), w mu (phi +- psi) with
// psi = A phi + g, so that psi takes two vectors A w, A w mu and g.  The way down then
// stores W, f, these two and g (108 doubles a layer at 16 streams) where the general
// form stores G, H and r (136) and reads them and the layer record (188) again on the
// way up; one product with W per layer, from registers, takes the place of six
// matrix-vector products in a chain.  Two more h^3 products per layer pay for it:
// 60,000 columns of 40 layers at 4 streams 0.80 -> 0.55 ms, 20,000 of 60 at 16 streams
// 1.89 -> 1.51 ms, one of 60 layers 240 -> 211 us (now 0.56 ms, 1.40 ms, 199 us).  With 32
// streams the products cost
// what the way up gains (its share of a layer is 20 %, 11 % at 64).
//
// Mapping: lane j of a team owns column j; products read the other operand from
// shared memory as broadcasts (one 16-byte word of each team per instruction),
// the inverses are symmetric sweeps whose pivot row is exchanged through shared
// memory.  A warp holds 32/TEAM instances and runs them in lockstep over its
// deepest column.  The layer record of the next layer is brought in with
// cp.async as soon as the current one's matrices are used up.
#pragma once

#include "dsp_device.cuh"

namespace dsp {

template <int N>
struct BCfg {
  static constexpr int H = N / 2;
  static constexpr int HP = mod_hp(N);          // row length of the records, even
  static constexpr int TEAM = pow2ceil(H);
  static constexpr int TPW = 32 / TEAM;         // instances per warp (= per CTA)
  // row stride of the matrices in shared memory: an odd number of 16-byte words,
  // so that 8 lanes reading one row each with 16-byte loads meet no conflict
  static constexpr int LDM = HP % 4 == 2 ? HP : HP + 2;
  static constexpr int MAT = H * LDM;
  static constexpr int NV = 7 * HP + 2;         // vectors of a layer record
  static constexpr int SB = 2 * HP + 4;         // pivot-row buffer of a sweep
  // team shared memory (doubles)
  static constexpr int O_X = 0;                 // X^T: row c = column c of X
  static constexpr int O_Y = O_X + MAT;         // Y^T
  static constexpr int O_A = O_Y + MAT;         // admittance A; up: H
  static constexpr int O_W = O_A + MAT;         // work; up: G
  static constexpr int O_V = O_W + MAT;         // layer-record vectors
  static constexpr int O_S = O_V + NV;          // 2 pivot-row buffers
  static constexpr int O_G = O_S + 2 * SB;      // gathered vectors, HP each:
  static constexpr int NG = 9;                  // g, w1, w2, gamma, scale, E / phi, D / w, w mu, d
  static constexpr int SIZE = O_G + NG * HP;
  // start of a team: the teams of a half warp are the width of a row apart, so that
  // their column reads (8 bytes a lane) fill the banks once, and the two halves 4 banks
  // apart, so that the broadcasts (16 bytes a team) do not meet either
  // (20,000 x 60 layers x 16 streams with all teams 4 banks apart 1.51 ms, so 1.38 ms);
  // STRIDE leaves room for the shift falling back between the halves
  static constexpr int HALF = TPW > 1 ? TPW / 2 : 1;
  static constexpr int STRIDE = (SIZE + (HALF - 1) * TEAM + 15) / 16 * 16;
  __device__ static constexpr int start(int team) {
    return team * STRIDE + team % HALF * TEAM + team / HALF * 2;
  }
  static_assert(NV % 2 == 0 && SB % 2 == 0 && TEAM % 2 == 0, "16-byte alignment");
  static constexpr size_t smem_bytes() { return sizeof(double) * (size_t)(TPW * STRIDE + (TPW > 1 ? 18 : 0)); }
  // resident warps per SM: as many as shared memory admits (228 KB, 1 KB reserved
  // per CTA), within 128 registers a thread at 16 warps and 255 at 8
  static constexpr int MINB_SMEM = (int)((228u * 1024u) / (smem_bytes() + 1024u));
  static constexpr int MINB_REGS = H <= 8 ? 16 : (H <= 16 ? 12 : 8);
  static constexpr int MINB = MINB_SMEM < MINB_REGS ? MINB_SMEM : MINB_REGS;
  static constexpr bool ROLL = H > 16;          // 64 streams: rolled outer loops
  // the lane's row of the identity in registers: diagonal elements as products
  // (the FP64 pipe has room) instead of selects by lane
  static constexpr bool IDREG = H <= 8;
  // fluxes without Jacobians: transmission records instead of G, H, r
  static constexpr bool LEAN = H <= 8;
};

// Negative inverse of a symmetric positive definite matrix with unit diagonal
// (the caller scales; +-1 in an indefinite one), columns held by the lanes: symmetric
// sweeps (Goodnight
// 1979, The American Statistician 33) of pivots 0..H-1.  In step k lane j's a[i]
// is row (k + i) mod H of its column: the update shifts it by one row, so every
// register index is a constant.  By symmetry the pivot column is the pivot row,
// one element per lane, exchanged through `buf` (twice, so that the rotated
// reads are contiguous; one double further in odd steps, to keep 16-byte
// alignment).  With a unit diagonal every pivot is <= 1, so the pivot lane can
// take the common update with 1 - 1/pivot in the place of the multiplier
// without losing digits: v - v (1 - p) = v p, p >= 1.
template <int H, int SB, bool CHECK>
__device__ __forceinline__ void sweep_step(double* a, const int j, const int k, const bool odd, const bool store,
                                           double* buf, bool& singular) {
  double* b = buf + (odd ? SB : 0);
  const int o = odd ? 1 : 0;
  if (store) {
    b[j + o] = a[0];
    b[j + H + o] = a[0];
  }
  __syncwarp();
  const double* v = b + k + o;
  const double d = v[0];
  double p = rcp_newton(d);
  if (CHECK && d == 0.0) {  // a zero pivot: its row and column are left out
    singular = true;
    p = 0.0;
  }
  const double c = a[0] * p;
  const double cc = j == k ? 1.0 - p : c;
  const double2* v2 = reinterpret_cast<const double2*>(v);
  {
    const double2 w = v2[0];
    if (H > 1) a[0] = fma(-cc, w.y, a[1]);
  }
#pragma unroll
  for (int i = 2; i < H; i += 2) {
    const double2 w = v2[i / 2];
    a[i - 1] = fma(-cc, w.x, a[i]);
    if (i + 1 < H) a[i] = fma(-cc, w.y, a[i + 1]);
  }
  a[H - 1] = j == k ? -p : c;
}

template <int H, int SB, bool ROLL, bool CHECK = false>
__device__ __forceinline__ void sweep_inverse(double* a, const int j, const bool store, double* buf, bool& singular) {
  if constexpr (ROLL) {
    static_assert(!ROLL || H % 2 == 0, "steps in pairs");
#pragma unroll 1
    for (int k = 0; k < H; k += 2) {
      sweep_step<H, SB, CHECK>(a, j, k, false, store, buf, singular);
      sweep_step<H, SB, CHECK>(a, j, k + 1, true, store, buf, singular);
    }
  } else {
#pragma unroll
    for (int k = 0; k < H; ++k) sweep_step<H, SB, CHECK>(a, j, k, (k & 1) != 0, store, buf, singular);
  }
  __syncwarp();
}

// sum_i a[i] v[i], v broadcast from shared memory (HP long, padded with 0)
template <int H>
__device__ __forceinline__ double dot_reg(const double* a, const double* v) {
  double s0 = 0.0, s1 = 0.0;
  const double2* v2 = reinterpret_cast<const double2*>(v);
#pragma unroll
  for (int i = 0; i < H; i += 2) {
    const double2 w = v2[i / 2];
    s0 = fma(a[i], w.x, s0);
    if (i + 1 < H) s1 = fma(a[i + 1], w.y, s1);
  }
  return s0 + s1;
}
// sum_i row[i] v[i], both in shared memory (row: this lane's own)
template <int H>
__device__ __forceinline__ double dot_row(const double* row, const double* v) {
  double s0 = 0.0, s1 = 0.0;
  const double2 *r2 = reinterpret_cast<const double2*>(row), *v2 = reinterpret_cast<const double2*>(v);
#pragma unroll
  for (int i = 0; i < H; i += 2) {
    const double2 x = r2[i / 2], w = v2[i / 2];
    s0 = fma(x.x, w.x, s0);
    if (i + 1 < H) s1 = fma(x.y, w.y, s1);
  }
  return s0 + s1;
}
// sum_i col[i * ld] v[i]: column `col` across the lanes
template <int H>
__device__ __forceinline__ double dot_col(const double* col, const int ld, const double* v) {
  double s0 = 0.0, s1 = 0.0;
  const double2* v2 = reinterpret_cast<const double2*>(v);
#pragma unroll
  for (int i = 0; i < H; i += 2) {
    const double2 w = v2[i / 2];
    s0 = fma(col[i * ld], w.x, s0);
    if (i + 1 < H) s1 = fma(col[(i + 1) * ld], w.y, s1);
  }
  return s0 + s1;
}
// acc[i] += M[k][i] f for one row k of a shared-memory matrix
template <int H>
__device__ __forceinline__ void axpy_row(double* acc, const double* row, const double f) {
  const double2* r2 = reinterpret_cast<const double2*>(row);
#pragma unroll
  for (int i = 0; i < H; i += 2) {
    const double2 m = r2[i / 2];
    acc[i] = fma(m.x, f, acc[i]);
    if (i + 1 < H) acc[i + 1] = fma(m.y, f, acc[i + 1]);
  }
}

// The instances of one warp: team `team` solves chunk slot `slot` (-1: none).
template <int N, bool GEN, bool SPH, bool LEAN, bool JAC = false>
__device__ __forceinline__ void bvp_warp(const FluxParams& p, const int slot) {
  using C = BCfg<N>;
  constexpr int H = C::H, HP = C::HP, TEAM = C::TEAM, LDM = C::LDM, SB = C::SB;
  constexpr bool ROLL = C::ROLL;
  constexpr double PI = 3.14159265358979323846;
  extern __shared__ double smem[];
  const int t = threadIdx.x % TEAM;
  const int j = t < H ? t : H - 1;  // lanes past the last column repeat it
  const bool own = t < H;
  double* const sm = smem + C::start(threadIdx.x / TEAM);
  double* const Xs = sm + C::O_X;
  double* const Ys = sm + C::O_Y;
  double* const As = sm + C::O_A;
  double* const Ws = sm + C::O_W;
  double* const vec = sm + C::O_V;
  double* const sbuf = sm + C::O_S;
  double* const vg = sm + C::O_G;
  double* const vw1 = vg + HP;
  double* const vw2 = vw1 + HP;
  double* const vgam = vw2 + HP;
  double* const vsc = vgam + HP;
  double* const ve = vsc + HP;  // E going down, phi going up
  double* const vd = ve + HP;
  double* const vwm = vd + HP;
  double* const vdp = vwm + HP;

  const bool ifb = (p.flags & DSP_FLAG_INDEX_FROM_BOTTOM) != 0;
  const int mrow = GEN ? (int)blockIdx.y : 0;
  const int m = GEN ? p.g.m + mrow : 0;
  // i: status / input / output index, L: layers, NT: output levels
  const int sl = slot >= 0 ? slot : 0;
  const int i = GEN ? p.g.ids[sl] : sl;
  const int L = GEN ? p.g.Ls[i] : p.L;
  const int NT = GEN ? (p.g.user_tau ? p.g.user_tau : L + 1) : L + 1;
  const InstLayout il = GEN ? InstLayout::make(L, N) : p.il;
  const double* const rec = p.inst_rec + (GEN ? p.g.inst_off[sl] : (long long)i * p.il.stride);
  const long long lay0 = GEN ? p.g.lay_off[sl] : (long long)i * p.L;
  const long long lstride = GEN ? p.g.lstride : (long long)lrec_stride(N);
  const double* const lrec0 = p.layer_rec + (GEN ? mrow * p.g.ms_layer : 0ll) + lay0 * lstride;
  constexpr int BSTRIDE = LEAN ? (JAC ? tjac_stride(N) : trec_stride(N)) : brec_stride(N);
  double* const brec0 = p.bvp_rec + (GEN ? mrow * p.g.ms_bvp : 0ll) + lay0 * BSTRIDE;
  auto oidx = [&](int lev) {
    if constexpr (GEN) return (long long)i * p.g.ntau_out + (ifb ? NT - 1 - lev : lev);
    else return (long long)i * NT + (ifb ? L - lev : lev);
  };
  double* const* outp = GEN ? p.g.out_flux : p.out;
  const GenLayout gly = GenLayout::make(GEN ? L : 0, N, GEN ? NT : 0);
  bool act = slot >= 0;
  if (act) {
    const int st0 = p.status ? p.status[i] : 0;
    // (GEN: an eigensystem missing at a mode says nothing of the modes before it)
    const bool no_solution = st0 == DSP_ERR_INVALID_INPUT || (GEN ? rec[gly.eig] <= (double)m : st0 == DSP_ERR_EIGEN);
    if (no_solution) {
      const double qnan = __longlong_as_double(0x7ff8000000000000ll);
      if (m == 0)
        for (int lev = t; lev < NT; lev += TEAM)
          for (int f = 0; f < 8; ++f) outp[f][oidx(lev)] = qnan;
      act = false;
    }
  }
  if constexpr (GEN) {
    if (act && (m > (int)rec[H_NAZ] || rec[H_DONE] != 0.0)) act = false;
  }
  const int ncut = act ? (int)rec[H_NCUT] : 0;
  const int Lw = (int)__reduce_max_sync(0xffffffffu, (unsigned)ncut);
  if (Lw == 0) return;
  DSP_PHASE_BEGIN
  const bool lyrcut = act && rec[H_LYRCUT] != 0.0;
  // modes m > 0 carry the beam only (DisortSolver.cpp:1246-1250, 1693-1748)
  const bool thermal = (p.flags & DSP_FLAG_THERMAL) != 0 && m == 0;
  const bool dlbc = (p.flags & DSP_FLAG_DIFFUSION_LOWER_BC) != 0;
  const double fbeam = act ? rec[H_FBEAM] : 0.0, umu0 = act ? rec[H_UMU0] : 1.0;
  const bool beam = fbeam > 0.0;
  const double* const taus = rec + il.tau_s;
  const double* const btr = rec + il.btr;
  const double dj = p.tables[tab_dsim(N) + j];
  const double wd = own ? 0.5 * p.tables[tab_wt(N) + j] / dj : 0.0;  // w / (2 d) of stream j
  const double muj = p.tables[tab_mu(N) + j];
  const double rumu0 = beam ? 1.0 / umu0 : 0.0;
  bool singular = false;

  // the layer record of layer l: X^T and the vectors, Y^T
  auto load_x = [&](int l) {
    if (l < ncut) {
      const double* lr = lrec0 + (long long)l * lstride;
      team_copy_mat<TEAM, HP, H, LDM>(Xs, lr + mod_X(N), t);
      team_copy_vec<TEAM, C::NV>(vec, lr + mod_k(N), t);
    }
    cp_async_commit();
  };
  auto load_y = [&](int l) {
    if (l < ncut) team_copy_mat<TEAM, HP, H, LDM>(Ys, lrec0 + (long long)l * lstride + mod_Y(N), t);
    cp_async_commit();
  };
  // per-layer scalars, loaded one layer ahead: scaled depths and beam factors of
  // the two boundaries; going up also 1 - omega and the unscaled depths
  struct Scal { double t0, t1, b0, b1, w1, u0, u1; };
  auto load_s = [&](int l, bool up) {
    Scal s{0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (l >= 0 && l < ncut) {
      s.t0 = taus[l];
      s.t1 = taus[l + 1];
      if (beam) {
        s.b0 = btr[l];
        s.b1 = btr[l + 1];
      }
      if (up) {
        const int lin = ifb ? L - 1 - l : l;
        s.w1 = 1.0 - (GEN ? p.g.ssa[p.g.in_off[i] + lin] : p.ssa(i, lin));
        if (!GEN && beam) {
          s.u0 = rec[il.tauc + l];
          s.u1 = rec[il.tauc + l + 1];
        }
      }
    }
    return s;
  };
  // pseudo-spherical beam: the record [c1 | d1 | xba | Chapman factor] of layer l
  auto SR = [&](int l) { return p.sph + (GEN ? mrow * p.g.ms_sph : 0ll) + (lay0 + l) * sph_stride(N); };
  // lane j's particular solution (c, d) at scaled depth tau of layer l; `bt` the
  // beam factor there (computeBeamSourceSpherical's form when SPH)
  auto particular = [&](int l, double tau, double bt, double& c, double& d) {
    c = 0.0;
    d = 0.0;
    if (beam) {
      if constexpr (SPH) {
        const double* sr = SR(l < ncut ? l : 0);
        const double e = exp(-sr[sph_xba(N)] * tau);
        c = e * fma(sr[j], tau, vec[3 * HP + j]);
        d = e * fma(sr[H + j], tau, vec[4 * HP + j]);
      } else {
        c = vec[3 * HP + j] * bt;
        d = vec[4 * HP + j] * bt;
      }
    }
    if (thermal) {
      const double x0 = vec[7 * HP], x1 = vec[7 * HP + 1];
      c = fma(vec[5 * HP + j], fma(x1, tau, x0), c);
      d = fma(vec[6 * HP + j], x1, d);
    }
  };

  // ------------------------------------------------------------------- down
  load_x(0);
  load_y(0);
  Scal sc = load_s(0, false);
  // odd h: the pad element of every gathered vector and row stays 0
  if (own) {
    for (int r = 0; r < HP; ++r) As[j * LDM + r] = r == j ? 1.0 : 0.0;
    const double inc = m == 0 && act ? rec[H_FISOT] + rec[H_PTOP] : 0.0;
    vg[j] = -2.0 * dj * inc;
  }
  if (HP != H && t == 0)
    for (int v = 0; v < C::NG; ++v) vg[v * HP + H] = 0.0;
  if (LEAN && own) {
    vd[j] = wd;
    vwm[j] = wd * muj;
  }
  __syncwarp();

  double a[H], id[C::IDREG ? H : 1];
  if constexpr (C::IDREG) {
#pragma unroll
    for (int r = 0; r < H; ++r) id[r] = r == j ? 1.0 : 0.0;
  }
  for (int l = 0; l < Lw; ++l) {
    const bool on = l < ncut;
    const Scal s = sc;
    sc = load_s(l + 1, false);
    cp_async_wait<1>();
    __syncwarp();
    const double ex = vec[HP + j], fx = vec[2 * HP + j];
    double ct, dt_, cb, db;
    particular(l, s.t0, s.b0, ct, dt_);
    particular(l, s.t1, s.b1, cb, db);
    double pl0 = 0.0, pl1 = 0.0;  // Planck source at the top and the bottom
    double jc = 0.0, jd = 0.0;    // thermal (c, d) of a unit source
    if (JAC) {
      jc = vec[5 * HP + j];
      jd = vec[6 * HP + j];
    }
    if (LEAN && thermal) {
      pl0 = fma(vec[7 * HP + 1], s.t0, vec[7 * HP]);
      pl1 = fma(vec[7 * HP + 1], s.t1, vec[7 * HP]);
    }
    DSP_PHASE(0)
    // I + M = I + X^T A X, column j
    const double* xj = Xs + j * LDM;
    double diag = 0.0;
    {
      double tv[H];
#pragma unroll
      for (int r = 0; r < H; ++r) tv[r] = 0.0;
      if constexpr (ROLL) {
#pragma unroll 2
        for (int r = 0; r < H; ++r) axpy_row<H>(tv, As + r * LDM, xj[r]);
      } else {
#pragma unroll
        for (int r = 0; r < H; ++r) axpy_row<H>(tv, As + r * LDM, xj[r]);
      }
      if constexpr (ROLL) {
        __syncwarp();  // every lane is done with A
#pragma unroll 2
        for (int r = 0; r < H; ++r) As[r * LDM + j] = dot_reg<H>(tv, Xs + r * LDM);
        diag = 1.0 + As[j * LDM + j];
      } else {
#pragma unroll
        for (int r = 0; r < H; ++r) {
          a[r] = dot_reg<H>(tv, Xs + r * LDM);
          if constexpr (C::IDREG) {
            a[r] += id[r];
            diag = fma(a[r], id[r], diag);
          } else if (r == j) {
            a[r] += 1.0;
            diag = a[r];
          }
        }
      }
    }
    const double gam = dot_row<H>(xj, vg);
    const double s1 = rsqrt(fabs(diag));
    if (own) {
      vw1[j] = gam - dt_ - ct;
      vsc[j] = s1;
      ve[j] = ex;
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < H; ++r) {
      if constexpr (ROLL) a[r] = r == j ? copysign(1.0, diag) : As[r * LDM + j] * (s1 * vsc[r]);
      else a[r] *= s1 * vsc[r];
    }
    // X and the vectors are used up: the next layer's start loading
    if constexpr (!LEAN) load_x(l + 1);
    DSP_PHASE(1)
    sweep_inverse<H, SB, ROLL>(a, j, own, sbuf, singular);
    DSP_PHASE(2)
    double* const br = brec0 + (long long)(on ? l : 0) * BSTRIDE;
#pragma unroll
    for (int r = 0; r < H; ++r) {
      a[r] = -a[r] * (s1 * vsc[r]);
      if (!LEAN && on && own) br[brec_H(N) + r * HP + j] = a[r];
    }
    const double hv = dot_reg<H>(a, vw1);
    const double rj = ct + hv;
    if (!LEAN && on && own) br[brec_r(N) + j] = rj;
    const double q = ex * rj;
    double xh = 0.0;  // X (r - c_t)
    double dphi = 0.0;
    bool past = false;
    // for the Jacobians: R, and hv, X hv of a unit source's value at the top and slope
    double rr[JAC ? H : 1], hv0 = 0.0, hv2 = 0.0, xj0 = 0.0, xj2 = 0.0;
    if constexpr (LEAN) {
      // V = X H E, column j, into the place of A
      double v[H];
#pragma unroll
      for (int r = 0; r < H; ++r) v[r] = 0.0;
#pragma unroll
      for (int r = 0; r < H; ++r) axpy_row<H>(v, Xs + r * LDM, a[r]);
      if (own) vgam[j] = hv;
      if constexpr (JAC) {
        if (own) {
#pragma unroll
          for (int r = 0; r < H; ++r) Ws[j * LDM + r] = v[r];  // X H
          sbuf[j] = -jc;
          sbuf[HP + j] = -jd;
        }
        __syncwarp();
        hv0 = dot_reg<H>(a, sbuf);
        hv2 = dot_reg<H>(a, sbuf + HP);
#pragma unroll
        for (int r = 0; r < H; ++r) rr[r] = 0.0;
#pragma unroll
        for (int r = 0; r < H; ++r) axpy_row<H>(rr, Ws + r * LDM, Xs[r * LDM + j]);  // X H X^T
        __syncwarp();
        if (own) {
          sbuf[j] = hv0;
          sbuf[HP + j] = hv2;
        }
        __syncwarp();
        xj0 = dot_col<H>(Xs + j, LDM, sbuf);
        xj2 = dot_col<H>(Xs + j, LDM, sbuf + HP);
      }
      __syncwarp();
      xh = dot_col<H>(Xs + j, LDM, vgam);
      if (on && own) {
#pragma unroll
        for (int r = 0; r < H; ++r) As[j * LDM + r] = ex * v[r];
      }
      // below the absorption cut of a thermal column the boundary-value problem has no
      // beam (btr = 0), but the reference's fluxes there still add its particular
      // solution: X c to phi and Y d to psi of the bottom level
      if constexpr (!SPH) {
        const bool mine = on && thermal && beam && s.b1 == 0.0;
        past = __any_sync(0xffffffffu, mine);
        if (past) {
          const double fact = mine ? exp(-s.t1 * rumu0) : 0.0;
          __syncwarp();
          if (own) {  // (a column without a beam has no beam terms in its record)
            vgam[j] = mine ? vec[3 * HP + j] * fact : 0.0;
            vdp[j] = mine ? vec[4 * HP + j] * fact : 0.0;
          }
          __syncwarp();
          dphi = dot_col<H>(Xs + j, LDM, vgam);
        }
      }
      __syncwarp();
      load_x(l + 1);
    }
    // Z = (1 - E^2) + 2 E H E
    const double ex2 = 2.0 * ex;
    diag = 0.0;
#pragma unroll
    for (int r = 0; r < H; ++r) {
      a[r] *= ex2 * ve[r];
      if constexpr (C::IDREG) {
        a[r] = fma(fx, id[r], a[r]);
        diag = fma(a[r], id[r], diag);
      } else if (r == j) {
        a[r] += fx;
        diag = a[r];
      }
    }
    const double s2 = rsqrt(fabs(diag));
    __syncwarp();  // every lane has read the first scale
    if (own) {
      vsc[j] = s2;
      vw2[j] = q - cb;
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < H; ++r) a[r] *= s2 * vsc[r];
    DSP_PHASE(3)
    sweep_inverse<H, SB, ROLL>(a, j, own, sbuf, singular);
    DSP_PHASE(4)
#pragma unroll
    for (int r = 0; r < H; ++r) {
      a[r] = -a[r] * (s2 * vsc[r]);
      if (!LEAN && on && own) br[brec_G(N) + r * HP + j] = a[r];
    }
    const double y = dot_reg<H>(a, vw2);  // G (q - c_b)
    const double gb = cb + db + 2.0 * y;
    if (own) {
      vgam[j] = gb;
      if (LEAN) vw1[j] = y;
#pragma unroll
      for (int r = 0; r < H; ++r) Ws[j * LDM + r] = !LEAN && r == j ? fma(2.0, a[r], -1.0) : 2.0 * a[r];
    }
    cp_async_wait<1>();  // Y of this layer
    __syncwarp();
    // A' = Y (2 G - I) Y^T, column j; g' = Y gamma'.  (LEAN: 2 G first, I taken off last, as
    // W and R take 2 G, of which 2 G - I keeps no digits where E > 1, the modes of -k; A'
    // before W, whose products the next layer does not wait for: 1.47 -> 1.39 ms)
    {
      double tv[H];
#pragma unroll
      for (int r = 0; r < H; ++r) tv[r] = 0.0;
#pragma unroll(ROLL ? 2 : H)
      for (int r = 0; r < H; ++r) axpy_row<H>(tv, Ws + r * LDM, Ys[r * LDM + j]);
      const double gn = dot_col<H>(Ys + j, LDM, vgam);
      double f = 0.0;
      if constexpr (LEAN) {
        f = fma(2.0, dot_col<H>(As + j, LDM, vw1), -xh);
        if constexpr (JAC) {
          // unit sources: y = G (E (c_t + hv) - c_b), f = 2 V y - X hv, g' = Y (c_b + d + 2 y)
          double *const b0 = sbuf, *const b1 = b0 + HP, *const b2 = b1 + HP;
          if (own) {
            b0[j] = ex * (jc + hv0);
            b1[j] = -jc;
            b2[j] = ex * hv2;
          }
          __syncwarp();
          const double y0 = dot_reg<H>(a, b0), y1 = dot_reg<H>(a, b1), y2 = dot_reg<H>(a, b2);
          __syncwarp();
          if (own) {
            b0[j] = 2.0 * y0;
            b1[j] = 2.0 * y1;
            b2[j] = 2.0 * y2;
          }
          __syncwarp();
          const double f0 = dot_col<H>(As + j, LDM, b0) - xj0, f1 = dot_col<H>(As + j, LDM, b1),
                       f2 = dot_col<H>(As + j, LDM, b2) - xj2;
          __syncwarp();
          if (own) {
            b1[j] += jc;
            b2[j] += jd;
          }
          __syncwarp();
          if (on && own) {
            double2* const o = reinterpret_cast<double2*>(br + tjac_s(N) + 6 * j);
            o[0] = make_double2(f0, f1);
            o[1] = make_double2(f2, dot_col<H>(Ys + j, LDM, b0));
            o[2] = make_double2(dot_col<H>(Ys + j, LDM, b1), dot_col<H>(Ys + j, LDM, b2));
          }
          // R = X H X^T - V (2 G) V^T
          double gv[H];
#pragma unroll
          for (int r = 0; r < H; ++r) gv[r] = 0.0;
#pragma unroll
          for (int r = 0; r < H; ++r) axpy_row<H>(gv, Ws + r * LDM, As[r * LDM + j]);
#pragma unroll
          for (int r = 0; r < H; ++r) axpy_row<H>(rr, As + r * LDM, -gv[r]);
          if (on && own) {
#pragma unroll
            for (int r = 0; r < H; ++r) br[tjac_R(N) + r * HP + j] = rr[r];
          }
        }
      }
      double w[H];
#pragma unroll
      for (int r = 0; r < H; ++r) w[r] = 0.0;
      if constexpr (ROLL) {
        __syncwarp();  // every lane is done with the work matrix
#pragma unroll
        for (int r = 0; r < H; ++r) Ws[r * LDM + j] = tv[r];
#pragma unroll 2
        for (int r = 0; r < H; ++r) axpy_row<H>(w, Ys + r * LDM, Ws[r * LDM + j]);
      } else {
#pragma unroll
        for (int r = 0; r < H; ++r) axpy_row<H>(w, Ys + r * LDM, LEAN ? tv[r] - Ys[r * LDM + j] : tv[r]);
      }
      if constexpr (LEAN) {
        // column j of W
        double wt[H];
#pragma unroll
        for (int r = 0; r < H; ++r) wt[r] = 0.0;
#pragma unroll
        for (int r = 0; r < H; ++r) axpy_row<H>(wt, As + r * LDM, tv[r]);
        if (on && own) {
#pragma unroll
          for (int r = 0; r < H; ++r) br[r * HP + j] = wt[r];
        }
        if (on && own) {
          double2* const o = reinterpret_cast<double2*>(br + trec_v(N) + 4 * j);
          o[0] = make_double2(f, past ? gn + dot_col<H>(Ys + j, LDM, vdp) : gn);
          if (thermal && beam) br[trec_dphi(N) + j] = dphi;
          o[1] = make_double2(dot_reg<H>(w, vd), dot_reg<H>(w, vwm));
          if (j == 0) *reinterpret_cast<double2*>(br + trec_pl(N)) = make_double2(pl0, pl1);
        }
        __syncwarp();  // every lane is done with V
      }
      if (on && own) {
#pragma unroll
        for (int r = 0; r < H; ++r) As[j * LDM + r] = w[r];
        vg[j] = gn;
      }
    }
    __syncwarp();
    load_y(l + 1);
    DSP_PHASE(5)
  }
  cp_async_wait<0>();
  __syncwarp();
  // ----------------------------------------------------------------- surface
  // up = R down + src at the bottom, psi = A phi + g:
  // [(I - R) + (I + R) A] phi = 2 src - (I + R) g.
  const double* sft = nullptr;
  if constexpr (GEN)
    if (p.g.brdf && !lyrcut && !dlbc) sft = p.g.brdf + (long long)sl * brdf_stride(N, p.g.numu);
  const double alb = m == 0 && act && !lyrcut && !dlbc && !sft ? rec[H_ALB] : 0.0;
  double* const bl = brec0 + (long long)(ncut > 0 ? ncut - 1 : 0) * BSTRIDE;  // the last layer's record
  // pseudo-spherical beam: the reference reflects Z0 times the beam factor at the
  // user angles (DisortSolver.cpp:3180-3218), not the solution at that depth; the
  // difference, in the downward intensities at the bottom
  double ddn = 0.0;
  if constexpr (GEN && SPH) {
    double dc = 0.0, dd = 0.0;
    if (act && beam) {
      const double* sr = SR(ncut - 1);
      const double tau = taus[ncut], e = exp(-sr[sph_xba(N)] * tau), bt = btr[ncut];
      dc = vec[3 * HP + j] * bt - e * fma(sr[j], tau, vec[3 * HP + j]);
      dd = vec[4 * HP + j] * bt - e * fma(sr[H + j], tau, vec[4 * HP + j]);
    }
    if (own) {
      vw1[j] = dc;
      vw2[j] = dd;
    }
    __syncwarp();
    ddn = 0.5 * (dot_col<H>(Xs + j, LDM, vw1) - dot_col<H>(Ys + j, LDM, vw2)) / dj;
    __syncwarp();
  }
  {
    // lane j's surface source (setMatrix :909-958, solve0 :993-1076)
    double src = 0.0;
    if (act) {
      const double fisob = m == 0 ? rec[H_FISOB] : 0.0, pbot = m == 0 ? rec[H_PBOT] : 0.0;
      if (dlbc) {
        src = pbot + p.tables[tab_mu(N) + j] * (m == 0 ? rec[H_PBOTD] : 0.0);
      } else {
        const double* srow = sft ? sft + j * brdf_row(N) : nullptr;
        if (!lyrcut && beam) src += (srow ? srow[0] : alb) * umu0 * fbeam * btr[ncut] / PI;
        src += fisob;
        if (thermal) src += (srow ? srow[H + 1] : 1.0 - alb) * pbot;
      }
    }
    const double sh = dj * src;
    if (own) {
      vw1[j] = sh;
      vw2[j] = dj;
    }
    __syncwarp();
    double rhs;
    if (!__any_sync(0xffffffffu, sft != nullptr)) {
      // Lambertian: (I + R)^{-1} (I - R) = I - 4 alb/(1 + alb) d d^T, so the
      // system is symmetric positive definite
      const double f = alb / (1.0 + alb);
      double dsrc = 0.0, diag = 0.0;
#pragma unroll
      for (int r = 0; r < H; ++r) {
        dsrc = fma(vw2[r], vw1[r], dsrc);
        a[r] = As[j * LDM + r] - 4.0 * f * dj * vw2[r];
        if (r == j) {
          a[r] += 1.0;
          diag = a[r];
        }
      }
      rhs = 2.0 * (sh - 2.0 * f * dj * dsrc) - vg[j];
      const double s1 = rsqrt(fabs(diag));
      __syncwarp();
      if (own) {
        vsc[j] = s1;
        vw1[j] = rhs;
      }
      __syncwarp();
#pragma unroll
      for (int r = 0; r < H; ++r) a[r] = r == j ? copysign(1.0, diag) : a[r] * (s1 * vsc[r]);
      sweep_inverse<H, SB, ROLL, true>(a, j, own, sbuf, singular);
#pragma unroll
      for (int r = 0; r < H; ++r) {
        a[r] = -a[r] * (s1 * vsc[r]);
        if ((!LEAN || JAC) && act && own) bl[(JAC ? tjac_inv(N) : brec_inv(N)) + r * HP + j] = a[r];
      }
    } else {
      // bidirectional surface: R_rc = (1 + delta_m0) d_r rho_rc d_c, not
      // symmetric in general; Gauss-Jordan inverse with row pivoting, column j
      // of [B | I] in the lane (B in shared memory for the pivot search)
      const double cpl = m == 0 ? 2.0 : 1.0;
      auto R = [&](int r, int c) { return sft ? cpl * vw2[r] * sft[r * brdf_row(N) + 1 + c] * vw2[c] : 0.0; };
      rhs = 2.0 * sh - vg[j];
      for (int c = 0; c < H; ++c) rhs -= R(j, c) * vg[c];
      for (int r = 0; r < H; ++r) {
        double v = As[r * LDM + j] + (r == j ? 1.0 : 0.0) - R(r, j);
        for (int c = 0; c < H; ++c) v = fma(R(r, c), As[c * LDM + j], v);
        if (own) Ws[r * LDM + j] = v;
      }
      __syncwarp();
      if (own)
        for (int r = 0; r < H; ++r) Xs[r * LDM + j] = r == j ? 1.0 : 0.0;
      if (own) vw1[j] = rhs;
      __syncwarp();
      for (int k = 0; k < H; ++k) {
        // the largest |B[r][k]|, r >= k (every lane runs the same search)
        int pr = k;
        double best = fabs(Ws[k * LDM + k]);
        for (int r = k + 1; r < H; ++r) {
          const double v = fabs(Ws[r * LDM + k]);
          if (v > best) {
            best = v;
            pr = r;
          }
        }
        __syncwarp();
        if (own && pr != k) {
          const double w0 = Ws[k * LDM + j], x0 = Xs[k * LDM + j];
          Ws[k * LDM + j] = Ws[pr * LDM + j];
          Ws[pr * LDM + j] = w0;
          Xs[k * LDM + j] = Xs[pr * LDM + j];
          Xs[pr * LDM + j] = x0;
        }
        __syncwarp();
        const double d = Ws[k * LDM + k];
        if (d == 0.0) singular = true;
        const double pv = d == 0.0 ? 0.0 : 1.0 / d;
        const double wk = Ws[k * LDM + j] * pv, xk = Xs[k * LDM + j] * pv;
        // columns <= k of B are finished (unit columns); the others and the inverse update
        for (int r = 0; r < H; ++r) {
          if (r == k) continue;
          const double f = Ws[r * LDM + k];
          if (own) {
            if (j > k) Ws[r * LDM + j] -= f * wk;
            Xs[r * LDM + j] -= f * xk;
          }
        }
        __syncwarp();
        if (own) {
          if (j > k) Ws[k * LDM + j] = wk;
          Xs[k * LDM + j] = xk;
        }
        __syncwarp();
      }
      // lane j: row j of the inverse (phi_j = sum_c Binv[j][c] rhs_c)
#pragma unroll
      for (int c = 0; c < H; ++c) {
        a[c] = Xs[j * LDM + c];
        if (!LEAN && act && own) bl[brec_inv(N) + c * HP + j] = a[c];
      }
    }
    __syncwarp();
    const double phi = dot_reg<H>(a, vw1);
    if (own) ve[j] = phi;
    __syncwarp();
    // downward intensities at the bottom, for the reflected field at the user angles
    if constexpr (GEN) {
      const double psi = dot_row<H>(As + j * LDM, ve) + vg[j];
      if (act && own) bl[brec_dn(N) + j] = 0.5 * (phi - psi) / dj + ddn;
    }
    __syncwarp();
  }
  DSP_PHASE(6)

  // --------------------------------------------------------------------- up
  bool nonfinite = false;
  // the eight outputs of a level from its angular sums (mean intensities su, sd, fluxes
  // fu, fd), the beam factor `fact` and the Planck source
  auto level_out = [&](double (&o)[8], double su, double sd, double fu, double fd, double fact, double ch,
                       double utau, double w1, double plsorc) {
    double dirint = 0.0, fldir = 0.0, fdir = 0.0;
    if (beam) {
      dirint = fbeam * fact;
      fldir = umu0 * fbeam * fact;
      fdir = SPH ? fabs(umu0) * fbeam * exp(-utau / ch) : umu0 * fbeam * exp(-utau * rumu0);
    }
    fu *= 2.0 * PI;
    fd *= 2.0 * PI;
    const double fdn = (fd + fldir) - fdir;
    constexpr double R4PI = 1.0 / (4.0 * PI);
    const double ua = 0.5 * (su + sd) + dirint * R4PI;
    const double uaso = dirint * R4PI;
    const double uad = 0.5 * sd, uau = 0.5 * su;
    const double dfdt = w1 * 4.0 * PI * (ua - plsorc);
    o[0] = fdir, o[1] = fdn, o[2] = fu, o[3] = dfdt, o[4] = ua, o[5] = uad, o[6] = uau, o[7] = uaso;
  };
  // fluxes at output level lu of layer l from the modal amplitudes (c, d) of the
  // homogeneous part there (computeFluxes, FluxSolver.cpp:1138-1287;
  // DisortSolver.cpp:1980-2124); `put`: this team has the level; `top`: the level is the
  // top of the column, where the downward intensities are the incoming ones (exactly: as
  // a difference of the modes they are rounding noise of the upward ones)
  const double incoming = act && m == 0 ? rec[H_FISOT] + rec[H_PTOP] : 0.0;
  auto eval_level = [&](int l, int lu, double utaupr, double utau, double w1, double c, double d, bool put, bool top) {
    const double ch = SPH && beam && put ? SR(l)[sph_ch(N)] : 1.0;
    const double fact = beam ? (SPH ? exp(-utaupr / ch) : exp(-utaupr * rumu0)) : 0.0;
    double cp, dp;
    particular(l, utaupr, fact, cp, dp);
    __syncwarp();
    if (own) {
      vgam[j] = c + cp;
      vd[j] = d + dp;
    }
    __syncwarp();
    const double ph = dot_col<H>(Xs + j, LDM, vgam), ps = dot_col<H>(Ys + j, LDM, vd);
    const double down = top ? 2.0 * dj * incoming : ph - ps, up = top ? 2.0 * ph - down : ph + ps;
    double su = wd * up, sd = wd * down;
    double fu = muj * su, fd = muj * sd;
#pragma unroll
    for (int off = TEAM / 2; off > 0; off >>= 1) {
      su += __shfl_xor_sync(0xffffffffu, su, off);
      sd += __shfl_xor_sync(0xffffffffu, sd, off);
      fu += __shfl_xor_sync(0xffffffffu, fu, off);
      fd += __shfl_xor_sync(0xffffffffu, fd, off);
    }
    if (put) {
      double o[8];
      level_out(o, su, sd, fu, fd, fact, ch, utau, w1, thermal ? fma(vec[7 * HP + 1], utaupr, vec[7 * HP]) : 0.0);
#pragma unroll
      for (int f = 0; f < 8; ++f)
        if ((f & (TEAM - 1)) == t) {
          outp[f][oidx(lu)] = o[f];
          if (!isfinite(o[f])) nonfinite = true;
        }
    }
  };
  const double* const utau_l = rec + gly.utau;
  const double* const utaus_l = rec + gly.utaus;
  const double* const lyr_l = rec + gly.lyr;
  // levels below the absorption cut carry zeros (computeFluxes :1151-1163;
  // DisortSolver.cpp:1998-2009)
  if constexpr (!GEN) {
    for (int lev = ncut + 1 + t; act && lev <= L; lev += TEAM)
      for (int f = 0; f < 8; ++f) outp[f][oidx(lev)] = 0.0;
  } else {
    if (m == 0)
      for (int lu = t; act && lu < NT; lu += TEAM)
        if ((int)lyr_l[lu] > ncut - 1)
          for (int f = 0; f < 8; ++f) outp[f][oidx(lu)] = 0.0;
  }
  if constexpr (LEAN) {
    // what the lane needs of layer l, loaded two layers ahead: row j of W, f, g, the
    // flux functionals of its bottom level
    struct Up { double2 w[HP / 2], fg, u; double dphi; };
    auto load_rec = [&](int l) {
      Up q{};
      if (l >= 0 && l < ncut) {
        const double* br = brec0 + (long long)l * BSTRIDE;
        const double2* row = reinterpret_cast<const double2*>(br + j * HP);
#pragma unroll
        for (int k = 0; k < HP / 2; ++k) q.w[k] = row[k];
        const double2* v = reinterpret_cast<const double2*>(br + trec_v(N) + 4 * j);
        q.fg = v[0];
        if (own) q.u = v[1];
        if (thermal && beam) q.dphi = br[trec_dphi(N) + j];
      }
      return q;
    };
    // TEAM consecutive levels are put out together, one per lane: their sums (kept when
    // the sweep passes the level) and scalars, loaded a group ahead
    struct Lev { double t1, u1, w1, pl, ch; };
    auto load_lev = [&](int base) {
      const int lev = base + t, la = lev > 0 ? lev - 1 : 0;  // the layer above
      Lev v{0.0, 0.0, 0.0, 0.0, 1.0};
      if (base >= 0 && lev <= ncut && act) {
        v.w1 = 1.0 - p.ssa(i, ifb ? L - 1 - la : la);
        if (thermal) v.pl = brec0[(long long)la * BSTRIDE + trec_pl(N) + (lev > 0 ? 1 : 0)];
        if (beam) {
          v.t1 = taus[lev];
          v.u1 = rec[il.tauc + lev];
          if (SPH) v.ch = SR(la)[sph_ch(N)];
        }
      }
      return v;
    };
    const double wdm = wd * muj;
    double su = 0.0, sd = 0.0, fu = 0.0, fd = 0.0;
    Lev lev = load_lev(Lw & ~(TEAM - 1));
    // level lu from this lane's phi (+ dphi), with psi's part sum u phi + w g
    auto level = [&](int lu, double phi, double dphi, double g, double u0, double u1) {
      double p0 = wd * (phi + dphi), p1 = wdm * (phi + dphi), q0 = fma(u0, phi, wd * g), q1 = fma(u1, phi, wdm * g);
#pragma unroll
      for (int off = TEAM / 2; off > 0; off >>= 1) {
        p0 += __shfl_xor_sync(0xffffffffu, p0, off);
        p1 += __shfl_xor_sync(0xffffffffu, p1, off);
        q0 += __shfl_xor_sync(0xffffffffu, q0, off);
        q1 += __shfl_xor_sync(0xffffffffu, q1, off);
      }
      if ((lu & (TEAM - 1)) == t) {
        su = p0 + q0;
        sd = p0 - q0;
        fu = p1 + q1;
        fd = p1 - q1;
      }
      if ((lu & (TEAM - 1)) == 0) {
        if (act && lu + t <= ncut) {
          double o[8];
          const double fact = beam ? (SPH ? exp(-lev.t1 / lev.ch) : exp(-lev.t1 * rumu0)) : 0.0;
          level_out(o, su, sd, fu, fd, fact, lev.ch, lev.u1, lev.w1, lev.pl);
#pragma unroll
          for (int f = 0; f < 8; ++f) {
            outp[f][oidx(lu + t)] = o[f];
            if (!isfinite(o[f])) nonfinite = true;
          }
        }
        lev = load_lev(lu - TEAM);
      }
    };
    double phi = ve[j];
    // one layer from its record, which then takes the one two layers up (two of them in
    // turn: a register move would wait for the load)
    auto step = [&](int l, Up& c) {
      double* const buf = l & 1 ? vgam : ve;
      if (own) buf[j] = phi;
      __syncwarp();
      level(l + 1, phi, c.dphi, c.fg.y, c.u.x, c.u.y);
      double s0 = c.fg.x, s1 = 0.0;
#pragma unroll
      for (int k = 0; k < H; k += 2) {
        const double2 v = reinterpret_cast<const double2*>(buf)[k / 2];
        s0 = fma(c.w[k / 2].x, v.x, s0);
        if (k + 1 < H) s1 = fma(c.w[k / 2].y, v.y, s1);
      }
      if (l < ncut) phi = s0 + s1;
      c = load_rec(l - 2);
    };
    Up q = load_rec(Lw - 1), q2 = load_rec(Lw - 2);
    int l = Lw - 1;
    for (; l > 0; l -= 2) {
      step(l, q);
      step(l - 1, q2);
    }
    if (l == 0) step(0, q);
    // the top: A = I, g = -2 d (incoming)
    level(0, phi, 0.0, own ? -2.0 * dj * incoming : 0.0, wd, wdm);
    DSP_PHASE(9)
  } else {
  const int NTw = GEN && m == 0 ? (int)__reduce_max_sync(0xffffffffu, act ? (unsigned)NT : 0u) : 0;
  auto load_up = [&](int l, int what) {
    if (l >= 0 && l < ncut) {
      const double* lr = lrec0 + (long long)l * lstride;
      const double* br = brec0 + (long long)l * brec_stride(N);
      if (what == 0) {
        team_copy_mat<TEAM, HP, H, LDM>(Ys, lr + mod_Y(N), t);
        team_copy_mat<TEAM, HP, H, LDM>(Xs, lr + mod_X(N), t);
        team_copy_vec<TEAM, C::NV>(vec, lr + mod_k(N), t);
      } else {
        team_copy_mat<TEAM, HP, H, LDM>(Ws, br + brec_G(N), t);  // G
        team_copy_mat<TEAM, HP, H, LDM>(As, br + brec_H(N), t);  // H
      }
    }
    cp_async_commit();
  };
  load_up(Lw - 1, 0);
  load_up(Lw - 1, 1);
  sc = load_s(Lw - 1, true);
  double r_next = Lw - 1 < ncut && own ? brec0[(long long)(Lw - 1) * brec_stride(N) + brec_r(N) + j] : 0.0;
  for (int l = Lw - 1; l >= 0; --l) {
    const bool on = l < ncut;
    const Scal s = sc;
    const double rj = r_next;
    if (l > 0) {
      sc = load_s(l - 1, true);
      r_next = l - 1 < ncut && own ? brec0[(long long)(l - 1) * brec_stride(N) + brec_r(N) + j] : 0.0;
    }
    cp_async_wait<0>();
    __syncwarp();
    DSP_PHASE(7)
    const double ex = vec[HP + j];
    double ct, dt_, cb, db;
    particular(l, s.t0, s.b0, ct, dt_);
    particular(l, s.t1, s.b1, cb, db);
    const double chom_b = dot_row<H>(Ys + j * LDM, ve) - cb;  // homogeneous C at the bottom
    if (own) vw1[j] = fma(ex, rj, chom_b);
    __syncwarp();
    const double b = dot_col<H>(Ws + j, LDM, vw1);
    if (own) vw2[j] = ex * b;
    __syncwarp();
    const double c = fma(2.0, dot_col<H>(As + j, LDM, vw2), -rj);  // homogeneous C at the top
    // D_ = sg (E2 bb - E1 aa): for a mode of -k with the decaying exponentials of |k| and
    // amplitudes from C at the two boundaries (a and b themselves lose E in digits)
    double aa = c - ex * b, bb = b, ee = ex, sg = 1.0, fx = vec[2 * HP + j];
    if (vec[j] < 0.0) {
      const double x = vec[j] * (s.t1 - s.t0);
      ee = exp(x);
      fx = -expm1(2.0 * x);
      bb = fx > 0.1 ? (chom_b - ee * c) / fx : ex * aa;
      aa = fx > 0.1 ? (c - ee * chom_b) / fx : ex * b;
      sg = -1.0;
    }
    if (own) vw1[j] = c + ct;
    __syncwarp();
    // G and H are used up
    load_up(l - 1, 1);
    const double phi = dot_col<H>(Xs + j, LDM, vw1);
    DSP_PHASE(8)
    if constexpr (GEN) {
      if (on && own) {
        double* cc = p.g.cc + mrow * p.g.ms_cc + (lay0 + l) * N;
        cc[j] = bb;
        cc[H + j] = aa;
      }
      if (m == 0) {
        const double k = fabs(vec[j]);
        for (int lu = 0; lu < NTw; ++lu) {
          const bool put = on && lu < NT && (int)lyr_l[lu] == l;
          if (!__any_sync(0xffffffffu, put)) continue;
          const double tu = put ? utaus_l[lu] : s.t0, x1 = tu - s.t0, x2 = s.t1 - tu;
          const double e1 = exp(-k * x1), e2 = exp(-k * x2);
          // C inside the layer from its values at the two boundaries (no cancellation)
          double cu = c;
          if (fx > 0.0) cu = (c * (e1 * -expm1(-2.0 * k * x2)) + chom_b * (e2 * -expm1(-2.0 * k * x1))) / fx;
          eval_level(l, lu, tu, put ? utau_l[lu] : 0.0, s.w1, cu, sg * (e2 * bb - e1 * aa), put, l == 0 && x1 == 0.0);
        }
      }
    } else {
      eval_level(l, l + 1, s.t1, s.u1, s.w1, chom_b, sg * (bb - ee * aa), on, false);
      if (l == 0) eval_level(0, 0, s.t0, s.u0, s.w1, c, sg * (ee * bb - aa), on, true);
    }
    __syncwarp();
    if (on && own) ve[j] = phi;
    load_up(l - 1, 0);
    __syncwarp();
    DSP_PHASE(9)
  }
  cp_async_wait<0>();
  }  // !LEAN
  DSP_PHASE_END
  if (act) {
    if (singular && t == 0) {
      if (GEN && m > 0) lower_mode(const_cast<double*>(rec) + gly.sing, m);
      else set_status(p.status, i, DSP_ERR_SINGULAR);
    }
    if (nonfinite) set_status(p.status, i, DSP_ERR_NONFINITE);
  }
}

// One team per instance, in chunk-slot order.
// JAC (up to 16 streams): flux_jac_lean_kernel follows and reads its part of the records.
template <int N, bool GEN = false, bool SPH = false, bool JAC = false>
__global__ void __launch_bounds__(32, JAC ? 8 : BCfg<N>::MINB) flux_bvp_kernel(FluxParams p) {
  using C = BCfg<N>;
  const int slot = blockIdx.x * C::TPW + threadIdx.x / C::TEAM;
  bvp_warp<N, GEN, SPH, !GEN && C::LEAN, JAC>(p, slot < p.n ? slot : -1);
}

// Persistent form (general solver): a resident grid whose warps take chunk slots
// from a work queue -- `order`, the chunk's slots by descending layer count (the
// size classes), consumed through one counter per mode -- so that the longest
// instances start first, the instances of a warp have about the same depth and
// the tail of the launch is short.
template <int N, bool SPH = false>
__global__ void __launch_bounds__(32, BCfg<N>::MINB) gen_bvp_persistent_kernel(FluxParams p, const int* order, int* heads) {
  using C = BCfg<N>;
  int* const head = heads + blockIdx.y;  // one queue per mode of the launch
  for (;;) {
    int k = 0;
    if (threadIdx.x == 0) k = atomicAdd(head, C::TPW);
    k = __shfl_sync(0xffffffffu, k, 0);
    if (k >= p.n) break;
    k += threadIdx.x / C::TEAM;
    bvp_warp<N, true, SPH, false>(p, k < p.n ? order[k] : -1);
    __syncwarp();  // the shared memory serves the next instances
  }
}

}  // namespace dsp
