"""GPU tests of the modal boundary-value kernel (csrc/flux_bvp.cuh) and the layer
records it reads, where their shapes have edges: instance counts that leave
teams of a warp empty, one to a few layers, every stream count (odd half counts
are padded), layers of zero and of very large optical depth, no scattering and
conservative scattering.

Tolerances: the flux parity of tests/parity.py (1e-9 relative, 1e-12 absolute)
against the extended-precision oracle.  At omega = 1 the oracle's own noise is
1e-8 (one eigenvalue is zero to rounding), so there the physics is the checker:
without absorption or emission the net flux is the same at every level, to a few
hundred rounding units of the flux scale (1e-13 x the incoming flux).
"""
import numpy as np
import pytest

import gpu_lib
import oracle_lib
from disort_b200 import capi, workloads
from parity import assert_parity

pytestmark = pytest.mark.gpu


def columns(N, n, L, seed, thermal, ssa=None):
    rng = np.random.default_rng(seed)
    dtau = np.clip(rng.lognormal(-2.0, 2.0, (n, L)), 1e-6, 20.0)
    om = rng.uniform(0.0, 0.99, (n, L)) if ssa is None else np.full((n, L), ssa)
    if ssa is None:
        dtau[:, L // 2] = 0.0        # an empty layer
        om[:, 0] = 0.0               # no scattering
        dtau[n // 2, L - 1] = 200.0  # opaque
    pc = N + 1
    arrays = dict(wavenumber_low=rng.uniform(300.0, 900.0, n), delta_tau=dtau, single_scat_albedo=om,
                  phase_function_moments=workloads.hg_moments(rng.uniform(-0.3, 0.85, (n, L)), pc),
                  temperature=200.0 + 90.0 * rng.random(L + 1), surface_albedo=rng.uniform(0.0, 1.0, n),
                  emissivity_top=0.7, direct_beam_flux=2.0, direct_beam_mu=rng.uniform(0.15, 0.95, n),
                  isotropic_flux_top=0.3, isotropic_flux_bottom=0.1, temperature_top=150.0, temperature_bottom=290.0)
    arrays["wavenumber_high"] = arrays["wavenumber_low"] + 5.0
    return dict(n_inst=n, num_streams=N, num_layers=L, num_phase_func_moments=0, pmom_count=pc,
                flags=capi.FLAG_THERMAL if thermal else 0, arrays=arrays)


@pytest.mark.parametrize("N", capi.SUPPORTED_NSTR)
@pytest.mark.parametrize("n,L", [(1, 1), (3, 2), (5, 7), (33, 3)])
def test_partial_warps_and_extreme_layers(N, n, L):
    for thermal in (True, False):
        w = columns(N, n, L, 100 * N + 10 * n + L, thermal)
        got, gst, rc = gpu_lib.flux_solve(w)
        ref, rst = oracle_lib.flux_solve(w, ext=True)
        assert rc == 0 and not gst.any() and not rst.any()
        assert_parity(got, ref, f"N={N} n={n} L={L} thermal={thermal}")


@pytest.mark.parametrize("N", [n for n in capi.SUPPORTED_NSTR if n <= 16])
@pytest.mark.parametrize("n,L", [(1, 1), (2, 8), (9, 17), (35, 40)])
def test_levels_below_the_absorption_cut(N, n, L):
    """Thermal columns with a beam, absorbing enough that the cut falls inside them: the
    boundary-value problem has no beam there, the fluxes still add its particular
    solution.  The two forms of the upward pass (fluxes alone, and before Jacobians)
    against the oracle; level groups of every length."""
    w = columns(N, n, L, 11 * N + n, True)
    w["arrays"]["delta_tau"] = np.where(w["arrays"]["delta_tau"] > 0, w["arrays"]["delta_tau"] * 4.0, 0.0)
    for extra in (0, capi.FLAG_INDEX_FROM_BOTTOM):
        got, gst, rc = gpu_lib.flux_solve(w, extra)
        jac = gpu_lib.flux_solve_jac(w, extra)
        ref, rst = oracle_lib.flux_solve(w, extra_flags=extra, ext=True)
        assert rc == 0 and not gst.any() and not rst.any()
        for form, out in (("fluxes", got), ("before Jacobians", jac[0])):
            # the divergence is 4 pi (1 - omega) (mean intensity - Planck): it has the
            # parity of the mean intensity, not of its own difference
            div = np.abs(out["flux_tau_divergence"] - ref["flux_tau_divergence"])
            assert (div <= 1e-9 * (4 * np.pi * ref["mean_intensity"] + np.abs(ref["flux_tau_divergence"])) + 1e-12).all()
            rest = dict(out, flux_tau_divergence=ref["flux_tau_divergence"])
            assert_parity(rest, ref, f"{form} N={N} n={n} L={L} flags={extra}")


@pytest.mark.parametrize("N", capi.SUPPORTED_NSTR)
def test_conservative_columns_conserve_the_net_flux(N):
    w = columns(N, 9, 12, 7 * N, False, ssa=1.0)
    got, gst, rc = gpu_lib.flux_solve(w)
    assert rc == 0 and not gst.any()
    net = got["flux_up"] - got["flux_down"] - got["flux_direct_beam"]
    incoming = np.pi * 0.3 + got["flux_direct_beam"][:, :1]
    assert np.max(np.abs(net - net[:, :1]) / incoming) <= 1e-13 * 300


@pytest.mark.parametrize("N", [4, 6, 8, 14, 16, 32, 64])
@pytest.mark.parametrize("which", [0, 1])
def test_indefinite_layers(N, which):
    """Layers whose phase moments make -A_s (an even moment far above 1) or -B_s (an
    odd one) indefinite: the eigensolver's other branch.  Unphysical but accepted,
    as by the oracle, which is the checker at its own double-extended distance
    (such columns amplify rounding)."""
    w = columns(N, 5, 3, 11 * N + which, True, ssa=0.9)
    w["arrays"]["delta_tau"] = np.clip(w["arrays"]["delta_tau"], 0.01, 0.5)
    pm = w["arrays"]["phase_function_moments"]
    pm[:, :, 1:] *= 0.2
    pm[::2, 1, 2 if which == 0 else 1] = 1.6
    got, gst, rc = gpu_lib.flux_solve(w)
    ref, rst = oracle_lib.flux_solve(w, ext=True)
    dbl, _ = oracle_lib.flux_solve(w)
    assert rc == 0 and np.array_equal(gst, rst)
    for f in capi.FLUX_OUT_FIELDS:
        spread = np.max(np.abs(dbl[f] - ref[f]) / (np.abs(ref[f]) + 1e-3))
        np.testing.assert_allclose(got[f], ref[f], rtol=1e-9 + 4.0 * spread, atol=1e-12 + 4e-3 * spread, err_msg=f)
