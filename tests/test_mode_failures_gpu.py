"""GPU tests of an azimuth mode that has no solution (neither -A_s nor -B_s positive
definite: unphysical moments, DSP_ERR_EIGEN), while the modes before it have.

The modes are solved several at a time (dsp_general.cu), but what an instance returns
is what the series taken mode by mode gives: the fluxes of mode 0 and the intensities
summed up to the mode before, both finite, with status EIGEN; and no error at all when
the convergence criterion ends the series before that mode is reached.  The instance's
neighbours in the batch are not touched.
"""
import numpy as np
import pytest

import gpu_lib
import oracle_lib
from disort_b200 import capi
from parity import assert_parity_general

pytestmark = pytest.mark.gpu

# stream count, first mode without a solution, omega and moments of the layer
CASES = [(4, 1, 0.542, [1.0, -0.083, 1.908, 2.526]),
         (8, 4, 0.848, [1.0, 0.013, 0.075, -0.076, -0.009, -0.091, 1.5, 1.014]),
         (14, 3, 0.874, [1.0, 0.324, 0.345, 0.172, 0.365, 0.254, -0.076, 0.171, -0.069, 1.181, 2.236, -2.383, -1.894,
                         -0.39])]


def batch(N, ssa, pm, broken, mu=(-0.7, 0.3), flags=0, accuracy=0.0):
    """Three 3-layer instances with a beam; the middle one has the layer `pm` when `broken`."""
    rng = np.random.default_rng(N)
    insts = []
    for k in range(3):
        moments = 0.6 ** np.arange(N + 1)[None, :] * np.ones((3, 1))
        moments[:, N] = 0.0  # no delta-M
        om = rng.uniform(0.2, 0.9, 3)
        if k == 1 and broken:
            moments[1, :N] = pm
            om[1] = ssa
        insts.append(dict(num_streams=N, num_layers=3, num_phase_func_moments=N, delta_tau=rng.uniform(0.1, 0.4, 3),
                          single_scat_albedo=om, phase_function_moments=moments, direct_beam_flux=1.0,
                          direct_beam_mu=0.55, surface_albedo=0.2, tau_user=[0.05, 0.15, 0.3], mu_user=list(mu),
                          phi_user=[0.0, 40.0, 130.0]))
    return capi.pack_general(insts, flags | capi.GFLAG_USER_TAU | capi.GFLAG_USER_MU, accuracy_fourier_series=accuracy)


def general_solve(d, persistent):
    ctx = gpu_lib.context()
    assert ctx.set_schedule([(N, 1, 1000000, 0, 0, persistent) for N in capi.SUPPORTED_NSTR]) == 0
    try:
        got, rc = gpu_lib.general_solve(d)
    finally:
        ctx.load_schedule_file(capi.TUNING_FILE)
    assert rc == 0
    return got


@pytest.mark.parametrize("persistent", [1, 2])
@pytest.mark.parametrize("N,first,ssa,pm", CASES)
def test_the_modes_before_it_stand(N, first, ssa, pm, persistent):
    got = general_solve(batch(N, ssa, pm, True), persistent)
    assert got["status"].tolist() == [0, capi.DSP_ERR_EIGEN, 0]
    well = general_solve(batch(N, ssa, pm, False), persistent)
    flux = general_solve(batch(N, ssa, pm, True, flags=capi.GFLAG_ONLY_FLUXES), persistent)
    assert not flux["status"].any()
    for f in capi.FLUX_OUT_FIELDS:
        np.testing.assert_array_equal(got[f], flux[f], err_msg=f)
        np.testing.assert_array_equal(got[f][::2], well[f][::2], err_msg=f)
    for f in ("intensity", "intensity_azimuth_avg"):
        np.testing.assert_array_equal(got[f][::2], well[f][::2], err_msg=f)
    # the oracle solves mode by mode and leaves the sum where it stopped
    ref = oracle_lib.general_solve(batch(N, ssa, pm, True), ext=True)
    assert ref["status"].tolist() == [0, capi.DSP_ERR_EIGEN, 0]
    assert np.isfinite(ref["intensity"]).all()
    assert_parity_general(got, ref, f"N={N}, modes below {first}")


@pytest.mark.parametrize("persistent", [1, 2])
def test_a_series_that_ends_before_it(persistent):
    """Near the vertical the terms fall by (1 - mu^2)^(1/2) ~ 5e-4 a mode: the series has
    converged to 5 % after modes 1 and 2, and mode 3, which has no solution, is solved in
    the same launch."""
    N, first, ssa, pm = CASES[2]
    d = batch(N, ssa, pm, True, mu=(-0.9999999, 0.9999999), accuracy=0.05)
    got = general_solve(d, persistent)
    ref = oracle_lib.general_solve(d, ext=True)
    assert not ref["status"].any() and not got["status"].any()
    assert_parity_general(got, ref, "converged")


@pytest.mark.parametrize("spherical", [False, True])
@pytest.mark.parametrize("N", capi.SUPPORTED_NSTR)
def test_every_form_of_the_boundary_value_kernel(N, spherical):
    """Every stream count in the per-instance and the persistent form, with a plane and a
    pseudo-spherical beam: the same bits; the plane beam also by the oracle's parity (the
    spherical source's own linear system is ill-conditioned: the oracle's double and
    extended builds differ by up to 2e-9 here, and tests/test_general_gpu.py holds it)."""
    rng = np.random.default_rng(7 * N + spherical)
    insts = []
    for k in range(40 if N <= 16 else 9):
        L = int(rng.integers(1, 9))
        dtau = rng.uniform(0.02, 0.6, L)
        insts.append(dict(num_streams=N, num_layers=L, num_phase_func_moments=N, delta_tau=dtau,
                          single_scat_albedo=rng.uniform(0.1, 0.95, L),
                          phase_function_moments=0.7 ** np.arange(N + 1)[None, :] * np.ones((L, 1)),
                          direct_beam_flux=1.0, direct_beam_mu=float(rng.uniform(0.2, 0.9)), surface_albedo=0.3,
                          temperature=220.0 + 60.0 * rng.random(L + 1), wavenumber_low=600.0, wavenumber_high=610.0,
                          temperature_bottom=285.0, level_altitudes=np.linspace(40.0, 0.0, L + 1),
                          bottom_radius=6371.0, tau_user=[0.0, float(dtau.sum()) / 3.0], mu_user=[-0.6, 0.2, 0.8],
                          phi_user=[0.0, 75.0]))
    flags = capi.GFLAG_USER_TAU | capi.GFLAG_USER_MU | capi.FLAG_THERMAL | (capi.FLAG_SPHERICAL_BEAM if spherical else 0)
    d = capi.pack_general(insts, flags)
    queue, each = general_solve(d, 1), general_solve(d, 2)
    assert not each["status"].any()
    for f in each:
        np.testing.assert_array_equal(queue[f], each[f], err_msg=f)
    if not spherical:
        assert_parity_general(each, oracle_lib.general_solve(d, ext=True), f"N={N}")
