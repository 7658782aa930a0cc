// gen_kernels.cuh — the general solver's own kernels (DisortSolver::solve):
// per-instance setup and the user-angle intensities of one azimuth mode.
//
// The per-layer eigensystems and particular solutions (flux_layer.cuh) and the
// boundary-value problem (flux_bvp.cuh) are shared with the flux solver; these kernels add what only the general solver has:
// ragged layer counts, user optical depths, the azimuth-mode schedule and
// intensities at user polar angles and azimuths.
#pragma once

#include "dsp_device.cuh"
#include "flux_layer.cuh"
#include "flux_setup.cuh"

namespace dsp {

// Setup of one instance per warp (disortSet, DisortSolver.cpp:641-866, and the
// decisions of DisortSolver::solve, :21-234).  Validation follows
// DisortConfig::validate (DisortConfig.cpp:72-249).
static __global__ void __launch_bounds__(128) gen_setup_kernel(FluxParams p) {
  __shared__ double stage[4][96];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = blockIdx.x * 4 + warp;
  if (slot >= p.n) return;
  const GenView& g = p.g;
  const int i = g.ids[slot];
  const int N = p.N, L = g.Ls[i];
  const int NT = g.user_tau ? g.user_tau : L + 1;
  const GenLayout gly = GenLayout::make(L > 0 ? L : 0, N, NT > 0 ? NT : 0);
  const InstLayout& il = gly.il;
  double* rec = p.inst_rec + g.inst_off[slot];
  const uint32_t fl = p.flags;
  const bool thermal = (fl & DSP_FLAG_THERMAL) != 0;
  const bool dlbc = (fl & DSP_FLAG_DIFFUSION_LOWER_BC) != 0;
  const bool ifb = (fl & DSP_FLAG_INDEX_FROM_BOTTOM) != 0;
  const bool only_fluxes = (fl & DSP_GFLAG_ONLY_FLUXES) != 0;
  const bool user_mu = (fl & DSP_GFLAG_USER_MU) != 0;
  const double fbeam = p.fbeam(i), umu0 = p.umu0(i), alb = p.alb(i), emis = p.emis(i);
  const double wlo = p.wlo(i), whi = p.whi(i), ttop = p.ttop(i), tbot = p.tbot(i);
  const int nmom = g.nmoms[i], pc = p.pc;
  const long long base = g.in_off[i];
  // index_from_bottom: inputs come bottom-up (reverseInputArrays, IndexConversion.hpp:16-40)
  auto dtau_at = [&](int lc) { return g.dtau[base + (ifb ? L - 1 - lc : lc)]; };
  auto ssa_at = [&](int lc) { return g.ssa[base + (ifb ? L - 1 - lc : lc)]; };
  auto pm_row = [&](int lc) { return g.pmom + (base + (ifb ? L - 1 - lc : lc)) * (long long)pc; };
  auto temp_at = [&](int lev) { return g.temp[base + i + (ifb ? L - lev : lev)]; };
  if (lane == 0) {
    for (int k = 0; k < 16; ++k) rec[k] = 0.0;
    rec[H_NT] = NT;
    rec[gly.eig] = kNoMode;
    rec[gly.sing] = kNoMode;
  }
  __syncwarp();  // other lanes store boundary Planck terms into the header below

  // ---- validate (DisortConfig.cpp:72-249) -------------------------------
  bool bad = L <= 0 || nmom < 0 || pc < (nmom > N ? nmom : N) + 1;
  if (!__any_sync(0xffffffffu, bad)) {
    for (int lc = lane; lc < L; lc += 32) {
      if (dtau_at(lc) < 0.0) bad = true;
      if (ssa_at(lc) < 0.0 || ssa_at(lc) > 1.0) bad = true;
    }
    if (thermal)
      for (int lev = lane; lev <= L; lev += 32)
        if (temp_at(lev) < 0.0) bad = true;
    if (user_mu) {
      const double* um = g.umu.row(i);
      for (int iu = lane; iu < g.numu_in; iu += 32) {
        if (fabs(um[iu]) > 1.0) bad = true;
        if (iu > 0 && um[iu] <= um[iu - 1]) bad = true;
      }
    }
    if (!only_fluxes) {
      const double* ph = g.phi.row(i);
      for (int j = lane; j < g.nphi; j += 32)
        if (ph[j] < 0.0 || ph[j] > 360.0) bad = true;
    }
    if (lane == 0) {
      if (thermal && (wlo < 0.0 || whi < wlo)) bad = true;
      if (dlbc && !thermal) bad = true;
      if (fbeam < 0.0) bad = true;
      if ((umu0 <= 0.0 || umu0 > 1.0) && fbeam > 0.0) bad = true;
      // the albedo is checked for a Lambertian surface only; a BRDF excludes the
      // diffusion lower boundary (DisortConfig.cpp:144-146, 160-163)
      if (g.brdf_type == DSP_BRDF_LAMBERTIAN && (alb < 0.0 || alb > 1.0)) bad = true;
      if (g.brdf_type != DSP_BRDF_LAMBERTIAN && dlbc) bad = true;
      if ((fl & DSP_FLAG_DELTA_M_PLUS) && nmom < N + 1) bad = true;
      // bottom_radius > 0 with the pseudo-spherical beam (DisortConfig.cpp:189-196)
      if ((fl & DSP_FLAG_SPHERICAL_BEAM) && !(p.rbot(i) > 0.0)) bad = true;
      if (thermal) {
        if (wlo < 0.0 || whi <= wlo) bad = true;
        if (ttop < 0.0 || tbot < 0.0) bad = true;
        if (emis < 0.0 || emis > 1.0) bad = true;
      }
    }
  }
  if (__any_sync(0xffffffffu, bad)) {
    if (lane == 0) set_status(p.status, i, DSP_ERR_INVALID_INPUT);
    return;
  }

  // ---- delta-M decisions (DisortSolver.cpp:72-112) ------------------------
  bool dm_local = false, dmp_fail = false;
  for (int lc = lane; lc < L; lc += 32) {
    const double pmN = pm_row(lc)[N];
    if (pmN != 0.0) dm_local = true;
    if (fl & DSP_FLAG_DELTA_M_PLUS) {
      const double pmN1 = pm_row(lc)[N + 1];
      if (pmN < 1e-4 || pmN1 < 0.7 * pmN) dmp_fail = true;
    }
  }
  bool deltam = __any_sync(0xffffffffu, dm_local);
  const bool dmplus = (fl & DSP_FLAG_DELTA_M_PLUS) && !__any_sync(0xffffffffu, dmp_fail);
  if (dmplus) deltam = false;

  // ---- per-layer scaling (disortSet, DisortSolver.cpp:663-747) -------------
  for (int lc = lane; lc < L; lc += 32) {
    const double w0 = ssa_at(lc), dt = dtau_at(lc);
    const double* pml = pm_row(lc);
    double f = 0.0, sig = 0.0, ws = w0, dts = dt, mode = 0.0;
    if (!deltam && !dmplus) {
      mode = 0.0;
    } else if (!dmplus || pml[N - 1] == pml[N] || pml[N] == pml[N + 1]) {
      f = pml[N];
      ws = w0 * (1.0 - f) / (1.0 - f * w0);
      dts = (1.0 - f * w0) * dt;
      mode = 1.0;
    } else {
      const double pmv = pml[N], pm1 = pml[N + 1];
      const double M = static_cast<double>(N);
      sig = ((M + 1.0) * (M + 1.0) - M * M) / (log(pmv * pmv) - log(pm1 * pm1));
      const double c = exp(M * M / (2.0 * sig));
      f = c * pmv;
      ws = w0 * (1.0 - f) / (1.0 - f * w0);
      dts = (1.0 - f * w0) * dt;
      mode = 2.0;
    }
    rec[il.dtau_s + lc] = dts;
    rec[il.ssa_s + lc] = ws;
    rec[il.fsc + lc] = f;
    rec[il.sig + lc] = sig;
    rec[il.mode + lc] = mode;
  }
  // Planck at the levels and the two boundaries (DisortSolver.cpp:186-202)
  if (thermal)
    for (int lev = lane; lev < L + 3; lev += 32) {
      const double B = planck2(wlo, whi, lev <= L ? temp_at(lev) : lev == L + 1 ? ttop : tbot, p.pk);
      if (lev <= L) rec[il.pkag + lev] = B;
      else if (lev == L + 1) rec[H_PTOP] = B * emis;
      else rec[H_PBOT] = B;
    }
  const SetupScan sc = setup_scan(rec, il, L, fbeam, umu0, stage[warp], lane, dtau_at, ssa_at);
  __syncwarp();

  if (lane == 0) {
    const bool lyrcut = (sc.total_abs >= 10.0 && !thermal && L > 1);
    const int ncut = lyrcut ? sc.ncut : L;
    double pbotd = 0.0;
    if (!thermal) {
      rec[H_PTOP] = 0.0;
      rec[H_PBOT] = 0.0;
    } else if (dlbc) {
      const double dl = rec[il.dtau_s + L - 1];
      if (dl > 0.0) pbotd = (rec[H_PBOT] - rec[il.pkag + L - 1]) / dl;
    }
    // highest azimuth mode (DisortSolver.cpp:218-234).  The reference reads
    // mu_user[1] and mu_user[2] (one past the index it means); entries past the
    // list count as 0 here.  Without intensities only mode 0 contributes.
    const int numu = (user_mu && !only_fluxes) ? g.numu_in : N;
    const double* um = (user_mu && !only_fluxes) ? g.umu.row(i) : nullptr;
    auto umu_at = [&](int k) { return (um && k < numu) ? um[k] : 0.0; };
    const bool indep = (fbeam == 0.0) || (fabs(1.0 - umu0) < 1.e-5) || only_fluxes ||
                       (numu == 1 && fabs(1.0 - umu_at(1)) < 1.e-5) ||
                       (numu == 1 && fabs(1.0 + umu_at(1)) < 1.e-5) ||
                       (numu == 2 && fabs(1.0 + umu_at(1)) < 1.e-5 && fabs(1.0 - umu_at(2)) < 1.e-5);
    const int naz = (indep || g.numu == 0) ? 0 : N - 1;
    rec[H_NCUT] = ncut;
    rec[H_LYRCUT] = lyrcut ? 1.0 : 0.0;
    rec[H_PBOTD] = pbotd;
    rec[H_DELTAM] = deltam ? 1.0 : 0.0;
    rec[H_DMPLUS] = dmplus ? 1.0 : 0.0;
    rec[H_FBEAM] = fbeam;
    rec[H_UMU0] = umu0;
    rec[H_ALB] = alb;
    rec[H_FISOT] = p.fisot(i);
    rec[H_FISOB] = p.fisob(i);
    rec[H_NAZ] = naz;
  }
  __syncwarp();
  // ---- output depths and their layers (DisortSolver.cpp:801-817) -----------
  const double total = rec[il.tauc + L];
  const double* ut_in = g.user_tau ? g.utau.row(i) : nullptr;
  for (int lu = lane; lu < NT; lu += 32) {
    double tau;
    if (ut_in) tau = ifb ? total - ut_in[NT - 1 - lu] : ut_in[lu];
    else tau = rec[il.tauc + lu];
    int lc;
    for (lc = 0; lc < L - 1; ++lc)
      if (tau >= rec[il.tauc + lc] && tau <= rec[il.tauc + lc + 1]) break;
    double tus = tau;
    if (deltam || dmplus) tus = rec[il.tau_s + lc] + (1.0 - ssa_at(lc) * rec[il.fsc + lc]) * (tau - rec[il.tauc + lc]);
    rec[gly.utau + lu] = tau;
    rec[gly.utaus + lu] = tus;
    rec[gly.lyr + lu] = lc;
  }
}

// P_l^m(-mu0) and P_l^m(mu_u) of mode m for every chunk slot (ptab): one thread
// per (slot, angle).
static __global__ void __launch_bounds__(128) gen_ptab_kernel(FluxParams p) {
  const GenView& g = p.g;
  const int na = 1 + g.numu;
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)p.n * na) return;
  const int slot = (int)(k / na), v = (int)(k % na);
  const int i = g.ids[slot];
  const double x = v == 0 ? -p.umu0(i) : g.umu.row(i)[v - 1];
  legendre_column(g.m + (int)blockIdx.y, x, p.N - 1, g.ptab + blockIdx.y * g.ms_ptab + k * p.N, 1);
}

// Eigenvectors and sources of every layer at the user polar angles for mode m
// (interpEigenvec, DisortSolver.cpp:2468-2504; interpSource, :2506-2580).  With
//   S_i, A_i = w_i / d_i sum_{l + m even, odd} g'_l / 2 P_l^m(mu_u) P_l^m(mu_i)
// (the two hemispheres differ in the sign of the odd terms) the intensity at mu_u
// scattered from the modes is (S X) C + (A Y) D, so that its coefficients of a
// and b are S X -/+ A Y.  A team of pow2ceil(h) lanes per layer task: lane i
// forms S_i, A_i, then lane j the products with row j of X^T and Y^T, which it
// keeps in registers over the angles.
template <int N>
struct ACfg {
  static constexpr int H = N / 2, HP = mod_hp(N), TEAM = pow2ceil(H), TPC = 128 / TEAM;
  static constexpr int TEAM_SMEM = N + 2 * HP;
};
template <int N>
__global__ void __launch_bounds__(128) gen_angle_kernel(FluxParams p) {
  using C = ACfg<N>;
  constexpr int H = C::H, HP = C::HP, TEAM = C::TEAM;
  __shared__ double smem[C::TPC * C::TEAM_SMEM];
  const int t = threadIdx.x % TEAM, j = t < H ? t : H - 1;
  const bool own = t < H;
  double* const gl = smem + (threadIdx.x / TEAM) * C::TEAM_SMEM;
  double* const sv = gl + N;
  double* const av = sv + HP;
  const unsigned msk = team_mask<TEAM>();
  const long long task = (long long)blockIdx.x * C::TPC + threadIdx.x / TEAM;
  if (task >= p.g.lay_off[p.n]) return;
  const LayerTask<N, true> q = layer_task<N, true>(p, task);
  if (!q.live) return;
  const int m = mode_of<true>(p), numu = p.g.numu;
  if (q.rec[task_layout<N>(p, q).eig] <= (double)m) return;
  const double ws = q.rec[q.il.ssa_s + q.lc];
  {
    const int mode = (int)q.rec[q.il.mode + q.lc];
    const double f = q.rec[q.il.fsc + q.lc], sig = q.rec[q.il.sig + q.lc];
    for (int k = t; k < N; k += TEAM) gl[k] = 0.5 * phase_coeff<true>(k, q.pml[k], mode, ws, f, sig);
  }
  if (HP != H && t == 0) {
    sv[H] = 0.0;
    av[H] = 0.0;
  }
  const double fbeam = q.rec[H_FBEAM];
  const bool beam = fbeam > 0.0, sph = (p.flags & DSP_FLAG_SPHERICAL_BEAM) != 0;
  const bool thermal = (p.flags & DSP_FLAG_THERMAL) && m == 0;
  double x[H], y[H];
#pragma unroll
  for (int r = 0; r < H; ++r) {
    x[r] = q.lrec[mod_X(N) + j * HP + r];
    y[r] = q.lrec[mod_Y(N) + j * HP + r];
  }
  // lane j's beam and thermal amplitudes (pseudo-spherical: the raw source at the
  // quadrature angles j, as the reference's interpSource reads it)
  double cb = 0.0, db = 0.0, ctv = 0.0, dtv = 0.0, xr0 = 0.0, xr1 = 0.0;
  if (beam) {
    cb = q.lrec[mod_cb(N) + j];
    db = q.lrec[mod_db(N) + j];
  }
  if (thermal) {
    ctv = q.lrec[mod_ct(N) + j];
    dtv = q.lrec[mod_dt(N) + j];
    xr0 = q.lrec[mod_xr(N)];
    xr1 = q.lrec[mod_xr(N) + 1];
  }
  const double dj = p.tables[tab_dsim(N) + j], wd = p.tables[tab_wt(N) + j] / dj;
  const double* const Y = p.tables + (long long)mode_row<true>() * tab_size(N) + tab_ylm(N);
  const double* const yb = beam_legendre<N, true>(p, q);
  const double fact = 2.0 * (m == 0 ? 1.0 : 2.0) * fbeam / (4.0 * 3.14159265358979323846);
  const int odd0 = 1 - (m & 1);  // first l of odd l + m
  double* const GU = q.lrec + glrec_gu(N);
  double* const zbu = GU + (long long)numu * N;
  __syncwarp(msk);
  for (int iu = 0; iu < numu; ++iu) {
    const double* pu = yb + (long long)N * (1 + iu);
    double se = 0.0, so = 0.0;
#pragma unroll 4
    for (int l = 0; l < N; l += 2) {
      se = fma(gl[l + 1 - odd0] * pu[l + 1 - odd0], Y[(l + 1 - odd0) * N + j], se);
      so = fma(gl[l + odd0] * pu[l + odd0], Y[(l + odd0) * N + j], so);
    }
    se *= wd;
    so *= wd;
    if (own) {
      sv[j] = se;
      av[j] = so;
    }
    __syncwarp(msk);
    double sx = 0.0, sy = 0.0;
#pragma unroll
    for (int r = 0; r < H; ++r) {
      sx = fma(x[r], sv[r], sx);
      sy = fma(y[r], av[r], sy);
    }
    if (own) {
      GU[(long long)iu * N + j] = sx + sy;
      GU[(long long)iu * N + H + j] = sx - sy;
    }
    // source terms: sums over the lanes
    double zb = 0.0, z0 = 0.0, z1 = 0.0;
    if (own) {
      if (beam) {
        zb = sph ? dj * (se * (cb + db) + so * (cb - db)) : sx * cb + sy * db;
        for (int l = j; l < N; l += H) zb = fma(gl[l] * pu[l], fact * yb[l], zb);
      }
      z0 = sx * ctv;
      z1 = sy * dtv;
    }
    if (beam || thermal) {
#pragma unroll
      for (int off = TEAM / 2; off > 0; off >>= 1) {
        zb += __shfl_xor_sync(msk, zb, off, TEAM);
        z0 += __shfl_xor_sync(msk, z0, off, TEAM);
        z1 += __shfl_xor_sync(msk, z1, off, TEAM);
      }
      if (t == 0) {
        if (beam) zbu[iu] = zb;
        if (thermal) {
          zbu[numu + iu] = fma(xr0, z0 + (1.0 - ws), xr1 * z1);
          zbu[2 * numu + iu] = xr1 * (z0 + (1.0 - ws));
        }
      }
    }
    __syncwarp(msk);
  }
}

// Intensities at the user angles for mode m (computeUserIntensities,
// DisortSolver.cpp:2938-3226): the formal solution along one user angle, layer by
// layer from the boundary the radiation comes from.  A team of pow2ceil(h) lanes
// per (slot, angle), lane j on eigenmode j: its share of the intensity at the
// layer's far side follows from the near side by I <- I exp(-dtau/|mu|) + (the
// layer's own), so every layer is passed once for all output depths, with one
// exponential and two reciprocals per lane; the lanes are summed only at the
// output depths (there with the part of the layer up to the depth).  I_m goes to
// imode; gen_fourier_kernel adds the modes up.
template <int N>
struct ICfg {
  static constexpr int H = N / 2, TEAM = pow2ceil(H), TPC = 128 / TEAM;
};
template <int N>
__global__ void __launch_bounds__(128) gen_intensity_kernel(FluxParams p) {
  using C = ICfg<N>;
  constexpr int H = C::H, TEAM = C::TEAM;
  constexpr double PI = 3.14159265358979323846;
  const GenView& g = p.g;
  const int t = threadIdx.x % TEAM, j = t < H ? t : H - 1;
  const bool own = t < H;
  const unsigned msk = team_mask<TEAM>();
  const int numu = g.numu;
  const long long item = (long long)blockIdx.x * C::TPC + threadIdx.x / TEAM;
  if (item >= (long long)p.n * numu) return;
  const int slot = (int)(item / numu), iu = (int)(item % numu);
  const int i = g.ids[slot];
  const int L = g.Ls[i];
  const int NT = g.user_tau ? g.user_tau : L + 1;
  const int mrow = (int)blockIdx.y, m = g.m + mrow;
  const int st0 = p.status ? p.status[i] : 0;
  if (st0 == DSP_ERR_INVALID_INPUT) return;
  const double* const rec = p.inst_rec + g.inst_off[slot];
  const GenLayout gly = GenLayout::make(L, N, NT);
  if (m > (int)rec[H_NAZ] || rec[H_DONE] != 0.0 || rec[gly.eig] <= (double)m) return;
  const InstLayout& il = gly.il;
  const int ncut = (int)rec[H_NCUT];
  const bool lyrcut = rec[H_LYRCUT] != 0.0;
  const bool thermal = (p.flags & DSP_FLAG_THERMAL) != 0 && m == 0;
  const bool dlbc = (p.flags & DSP_FLAG_DIFFUSION_LOWER_BC) != 0;
  const double fbeam = rec[H_FBEAM], umu0 = rec[H_UMU0];
  const bool beam = fbeam > 0.0;
  const double* const taus = rec + il.tau_s;
  const double* const btr = rec + il.btr;
  const double* const utaus = rec + gly.utaus;
  const double* const lyr = rec + gly.lyr;
  const double* const lrec0 = p.layer_rec + mrow * g.ms_layer + g.lay_off[slot] * g.lstride;
  const double* const cc0 = g.cc + mrow * g.ms_cc + g.lay_off[slot] * N;
  const double umv = g.umu.row(i)[iu];
  const bool neg = umv < 0.0;
  const double nu = fabs(umv);
  double* const out = g.imode + mrow * g.ms_int + (long long)slot * g.nt_max * numu + iu;
  auto total = [&](double v) {
#pragma unroll
    for (int off = TEAM / 2; off > 0; off >>= 1) v += __shfl_xor_sync(msk, v, off, TEAM);
    return v;
  };

  // boundary radiation at the angle (DisortSolver.cpp:3180-3226)
  double bnd = 0.0;
  if (neg) {
    if (m == 0) bnd = rec[H_FISOT] + rec[H_PTOP];
  } else if (dlbc) {
    if (!lyrcut && m == 0) bnd = rec[H_PBOT] + umv * rec[H_PBOTD];
  } else if (!lyrcut) {
    const double* const mu = p.tables + tab_mu(N);
    const double* const wt = p.tables + tab_wt(N);
    // the downward intensities at the bottom come with the boundary-value solution
    const double dfu = own ? p.bvp_rec[mrow * g.ms_bvp + (g.lay_off[slot] + ncut - 1) * brec_stride(N) + brec_dn(N) + j] : 0.0;
    const double muw = mu[j] * wt[j];
    if (g.brdf) {
      // bidirectional surface at user angles; the isotropic bottom flux enters at
      // every mode, as the reference adds it (DisortSolver.cpp:3213-3220)
      const double* ur = g.brdf + (long long)slot * brdf_stride(N, numu) + (H + iu) * brdf_row(N);
      const double refl = total((m == 0 ? 2.0 : 1.0) * ur[1 + j] * muw * dfu);
      bnd = refl + umu0 * fbeam / PI * ur[0] * btr[L] + (m == 0 ? ur[H + 1] * rec[H_PBOT] : 0.0) + rec[H_FISOB];
    } else if (m == 0) {
      // Lambertian surface at user angles: set for mu > 0 only (DisortSolver.cpp:2655-2662)
      const double alb = rec[H_ALB];
      const double refl = total(2.0 * muw * dfu);
      const double rho = umv > 0.0 ? alb : 0.0, em = umv > 0.0 ? 1.0 - alb : 0.0;
      bnd = rho * refl + umu0 * fbeam / PI * rho * btr[L] + em * rec[H_PBOT] + rec[H_FISOB];
    }
  }

  // output depths below the cut carry zeros
  for (int lu = t; lu < NT; lu += TEAM)
    if (lyrcut && (int)lyr[lu] >= ncut) out[(long long)lu * numu] = 0.0;
  const int my_lyr = t < NT ? (int)lyr[t] : -1;  // the first TEAM depths' layers, kept
  const double rnu = 1.0 / nu, rmu0 = beam ? 1.0 / umu0 : 0.0;
  const double bden = neg ? 1.0 - nu * rmu0 : 1.0 + nu * rmu0;
  const bool bres = fabs(bden) < 0.0001;
  const double rbden = bres ? 0.0 : 1.0 / bden;
  // lane j's share of the intensity, and the beam and thermal parts (every lane the same)
  // (accr: the beam's part at an angle that resonates with mu0, where the reference's
  // limit carries the attenuation of the output depth, DisortSolver.cpp:3010-3030)
  double acc = 0.0, accs = 0.0, accr = 0.0;
  for (int s = 0; s < ncut; ++s) {
    const int l = neg ? s : ncut - 1 - s;
    const double* const lr = lrec0 + (long long)l * g.lstride;
    const double* const gu = lr + glrec_gu(N) + (long long)iu * N;
    const double* const zu = lr + glrec_gu(N) + (long long)numu * N;
    const double* const x = cc0 + (long long)l * N;
    // (a mode of -k: the exponentials of |k|, with the signs of its D_, flux_bvp.cuh)
    const double kr = lr[mod_k(N) + j], k = fabs(kr), we = lr[mod_E(N) + j];
    const double g0 = own ? gu[j] : 0.0, g1 = own ? gu[H + j] : 0.0;
    const bool minus = kr < 0.0;
    const double wk = minus ? rcp_newton(we) : we;
    const double gb = (minus ? g1 : g0) * x[j], ga = (minus ? g0 : g1) * x[H + j];
    const double tt = taus[l], tb = taus[l + 1], dt = tb - tt;
    const double e = exp(-dt * rnu);
    const double t0 = neg ? tt : tb;  // the near side, where the radiation enters
    // the mode that grows towards the far side (down: a from the top; up: b from the
    // bottom) meets the resonance k = 1/|mu|
    const double gn = neg ? ga : gb, gf = neg ? gb : ga;
    const double den = 1.0 - nu * k;
    const bool res = fabs(den) < 0.0001;
    const double rn = res ? 0.0 : rcp_newton(den), rf = rcp_newton(1.0 + nu * k);
    const double b0 = beam ? btr[l] : 0.0, b1 = beam ? btr[l + 1] : 0.0;
    const double zb = beam ? zu[iu] : 0.0, z0 = thermal ? zu[numu + iu] : 0.0, z1 = thermal ? zu[2 * numu + iu] : 0.0;
    // output depths in this layer: the part of the layer on the boundary side
    for (int base = 0; base < NT; base += TEAM) {
      const int v = base == 0 ? my_lyr : (base + t < NT ? (int)lyr[base + t] : -1);
      unsigned hit = __ballot_sync(msk, v == l) >> (threadIdx.x & 31u & ~(unsigned)(TEAM - 1));
      if constexpr (TEAM < 32) hit &= (1u << TEAM) - 1u;
      while (hit) {
        const int lu = base + __ffs(hit) - 1;
        hit &= hit - 1u;
        const double ut = utaus[lu];
        const double d = neg ? ut - t0 : t0 - ut;  // depth from the near side
        double v1 = acc, v2 = accs, ed = 1.0;
        const double exp0 = beam ? exp(-ut * rmu0) : 0.0;
        if (bres) v2 += accr * exp0;
        if (fabs(d) >= 1e-6) {
          ed = exp(-d * rnu);
          // the near mode at the depth (1 at the near side), the far mode there and
          // at the near side (wk)
          const double en = exp(-k * d), ef = exp(-k * (neg ? tb - ut : ut - tt));
          v1 = acc * ed + gn * (res ? d * rnu * ed : (en - ed) * rn) + gf * ((ef - wk * ed) * rf);
          v2 = fma(accs, ed, bres ? accr * exp0 : 0.0);
          if (beam) v2 += zb * (bres ? d * rmu0 * exp0 : (exp0 - (neg ? b0 : b1) * ed) * rbden);
          if (thermal) v2 += z0 * (1.0 - ed) + z1 * ((ut + umv) - (t0 + umv) * ed);
        }
        const double dist = neg ? ut : taus[L] - ut;
        const double I = total(v1) + v2 + (bnd != 0.0 ? bnd * exp(-dist * rnu) : 0.0);
        if (t == 0) out[(long long)lu * numu] = I;
      }
    }
    // across the layer
    acc = acc * e + gn * (res ? dt * rnu * e : (wk - e) * rn) + gf * ((1.0 - wk * e) * rf);
    if (beam) {
      const double bn = neg ? b0 : b1, bf = neg ? b1 : b0;
      if (bres) accr = fma(zb, dt * rmu0, accr);
      accs = accs * e + zb * ((bf - bn * e) * rbden);  // (rbden is 0 at resonance)
    } else {
      accs *= e;
    }
    if (thermal) accs += z0 * (1.0 - e) + z1 * (((neg ? tb : tt) + umv) - (t0 + umv) * e);
  }
}

// The Fourier sum over the modes of a launch (DisortSolver.cpp:3228-3266), one
// warp per instance, a lane per (level, angle) pair; in mode order, with the
// azimuthal convergence test after each mode (:337-347), so that a mode past
// the convergence adds nothing even when it was computed with the others.  The series
// also ends at a mode that has no eigensystem, with the sum of the modes before it.
static __global__ void __launch_bounds__(128) gen_fourier_kernel(FluxParams p, int modes) {
  constexpr double PI = 3.14159265358979323846;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = blockIdx.x * 4 + warp;
  if (slot >= p.n) return;
  const GenView& g = p.g;
  const int i = g.ids[slot];
  const int L = g.Ls[i];
  const int NT = g.user_tau ? g.user_tau : L + 1;
  const int numu = g.numu, nphi = g.nphi, nk = NT * numu;
  const bool ifb = (p.flags & DSP_FLAG_INDEX_FROM_BOTTOM) != 0;
  auto elem = [&](int k) {
    const int lu = k / numu, iu = k % numu;
    return ((long long)i * g.ntau_out + (ifb ? NT - 1 - lu : lu)) * g.numu_out + iu;
  };
  const int st0 = p.status ? p.status[i] : 0;
  if (st0 == DSP_ERR_INVALID_INPUT || st0 == DSP_ERR_EIGEN) {
    if (g.m == 0) {
      const double qnan = __longlong_as_double(0x7ff8000000000000ll);
      for (int k = lane; k < nk; k += 32) {
        const long long o2 = elem(k);
        g.out_iavg[o2] = qnan;
        for (int j = 0; j < nphi; ++j) g.out_int[o2 * nphi + j] = qnan;
      }
    }
    return;
  }
  double* const rec = p.inst_rec + g.inst_off[slot];
  const int naz = (int)rec[H_NAZ];
  if (rec[H_DONE] != 0.0) return;
  const GenLayout gly = GenLayout::make(L, p.N, NT);
  const double eig = rec[gly.eig], sing = rec[gly.sing];
  double kconv = rec[H_KCONV];
  const double* const ph = g.phi.row(i);
  const double phi0 = g.phi0(i);
  for (int mi = 0; mi < modes; ++mi) {
    const int m = g.m + mi;
    if (m > naz) break;
    if (eig <= (double)m) {  // (mode 0: status EIGEN, above)
      __syncwarp();
      if (lane == 0) {
        set_status(p.status, i, DSP_ERR_EIGEN);
        rec[H_DONE] = 1.0;
      }
      return;
    }
    if (sing <= (double)m && lane == 0) set_status(p.status, i, DSP_ERR_SINGULAR);
    const double* const im = g.imode + mi * g.ms_int + (long long)slot * g.nt_max * numu;
    double maxr = 0.0;
    for (int j0 = 0; j0 < nphi || j0 == 0; j0 += 32) {
      const int nj = nphi - j0 < 32 ? nphi - j0 : 32;
      double cm = 1.0;
      if (m > 0 && lane < nj) cm = cos(static_cast<double>(m) * ((ph[j0 + lane] - phi0) * PI / 180.0));
      for (int kb = 0; kb < nk; kb += 32) {
        const int k = kb + lane;
        const double I = k < nk ? im[k] : 0.0;
        const long long o2 = k < nk ? elem(k) : 0;
        if (m == 0 && j0 == 0 && k < nk) g.out_iavg[o2] = I;
        for (int j = 0; j < nj; ++j) {
          const double az = I * __shfl_sync(0xffffffffu, cm, j);
          if (k >= nk) continue;
          double& acc = g.out_int[o2 * nphi + j0 + j];
          const double v = m == 0 ? az : acc + az;
          acc = v;
          const double uu = fabs(v);
          double ratio;
          if (uu == 0.0) ratio = 1.0 + fabs(az);
          else if (fabs(az) == 0.0) ratio = 0.0;
          else ratio = fabs(az) / uu;
          maxr = fmax(maxr, ratio);
        }
      }
    }
    if (m > 0 && g.accur > 0.0) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) maxr = fmax(maxr, __shfl_xor_sync(0xffffffffu, maxr, off));
      if (maxr <= g.accur) kconv += 1.0;
      if (kconv >= 2.0) {
        __syncwarp();
        if (lane == 0) {
          rec[H_KCONV] = kconv;
          rec[H_DONE] = 1.0;
        }
        return;
      }
    }
  }
  if (lane == 0) rec[H_KCONV] = kconv;
}

}  // namespace dsp
