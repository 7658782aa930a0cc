"""GPU tests of the general solver's mode batches: the azimuth modes of a chunk
run side by side as far as the workspace allows (dsp_general.cu), and every mode
is computed on its own, so the results do not depend on how many share a launch.

A smaller workspace (DSP_WORKSPACE_MB) cuts the batches and the chunks: outputs
must be bit-identical, with output depths at user optical depths and at the
levels, with more azimuths than lanes, and with the convergence criterion ending
the series inside a batch (checked against the oracle's sequential rule by the
parity test)."""
import numpy as np
import pytest

import gpu_lib
from disort_b200 import capi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nstr,levels,accur", [((4, 6), False, 0.0), ((16,), True, 0.0), ((14, 32), False, 0.0),
                                               ((64,), True, 0.0), ((8, 32), False, 1e-3)])
def test_results_do_not_depend_on_the_mode_batch(monkeypatch, nstr, levels, accur):
    rng = np.random.default_rng(5)
    insts = []
    for k in range(7 if 64 not in nstr else 3):
        N, L = nstr[k % len(nstr)], int(rng.integers(1, 40))
        dtau = np.clip(rng.lognormal(-2.0, 2.0, L), 1e-6, 20.0)
        insts.append(dict(num_streams=N, num_layers=L, num_phase_func_moments=N + 1, delta_tau=dtau,
                          single_scat_albedo=rng.uniform(0.0, 0.99, L),
                          phase_function_moments=workloads.hg_moments(rng.uniform(0.5, 0.95, L), N + 2),
                          direct_beam_flux=1.0, direct_beam_mu=float(rng.uniform(0.1, 0.95)), surface_albedo=0.3,
                          tau_user=[0.0, workloads.column_total(dtau) / 3.0], mu_user=[-0.8, -0.1, 0.4],
                          phi_user=list(np.linspace(0.0, 350.0, 37))))
    flags = capi.FLAG_DELTA_M_PLUS | capi.GFLAG_USER_MU | (0 if levels else capi.GFLAG_USER_TAU)
    d = capi.pack_general(insts, flags, accuracy_fourier_series=accur)
    got, rc = gpu_lib.general_solve(d)
    assert rc == 0 and not got["status"].any()
    monkeypatch.setenv("DSP_WORKSPACE_MB", "16")
    small, rc = gpu_lib.general_solve(d)
    assert rc == 0
    for f in got:
        np.testing.assert_array_equal(got[f], small[f], err_msg=f)


@pytest.mark.parametrize("offset", [0.0, 3e-5, -8e-5, 2e-4])
def test_user_angles_that_resonate_with_the_beam(offset):
    """Downward user angles within 1e-4 of -mu0 take the reference's limit of the
    beam term, others its closed form: general parity (1e-9, tests/parity.py)."""
    import oracle_lib
    from parity import assert_parity_general
    rng = np.random.default_rng(17)
    insts = []
    for k in range(6):
        N, L = (8, 16)[k % 2], int(rng.integers(2, 25))
        dtau = np.clip(rng.lognormal(-2.0, 1.5, L), 1e-4, 5.0)
        insts.append(dict(num_streams=N, num_layers=L, num_phase_func_moments=N + 1, delta_tau=dtau,
                          single_scat_albedo=rng.uniform(0.0, 0.95, L),
                          phase_function_moments=workloads.hg_moments(rng.uniform(0.3, 0.9, L), N + 2),
                          direct_beam_flux=1.0, direct_beam_mu=0.5 * (1.0 + offset), surface_albedo=0.2,
                          tau_user=[0.0, float(dtau[0]) / 3.0, workloads.column_total(dtau)], mu_user=[-0.5, 0.5],
                          phi_user=[0.0, 90.0]))
    d = capi.pack_general(insts, capi.FLAG_DELTA_M_PLUS | capi.GFLAG_USER_TAU | capi.GFLAG_USER_MU)
    got, rc = gpu_lib.general_solve(d)
    ref = oracle_lib.general_solve(d)
    ref = ref[0] if isinstance(ref, tuple) else ref
    assert rc == 0 and not got["status"].any()
    assert_parity_general(got, ref, f"offset {offset}")
