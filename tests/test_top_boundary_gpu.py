"""GPU test: what the boundary condition at the top says of the downward field.

With no diffuse radiation coming in, the downward diffuse flux and mean intensity at
optical depth 0 are zero, with isotropic radiation I they are pi I and I / 2 (half of
the sphere), whatever lies below.  Both forms of the boundary-value kernel have to
give them from the boundary condition, not as a difference of the layer's modes:
exactly zero in the one case, within the roundings of a sum over up to 32 streams and
its weights (64 units, with a beam also of its flux, which is added and taken out
again) in the other.  The same for the temperature derivatives of the two, which are
zero.
"""
import numpy as np
import pytest

import gpu_lib
from disort_b200 import capi, workloads

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def check_top(down, mean_down, incoming, direct=0.0):
    if incoming == 0.0:
        assert not down.any() and not mean_down.any()
    else:
        assert (np.abs(down - np.pi * incoming) <= 64 * EPS * (np.pi * incoming + direct)).all()
        assert (np.abs(mean_down - 0.5 * incoming) <= 64 * EPS * incoming).all()


@pytest.mark.parametrize("incoming", [0.0, 0.3])
@pytest.mark.parametrize("N", capi.SUPPORTED_NSTR)
def test_flux_path(N, incoming):
    w = workloads.thermal_sweep(n_bands=5, num_layers=7, num_streams=N, seed=N)
    w["arrays"].update(isotropic_flux_top=incoming, direct_beam_flux=0.0, emissivity_top=1.0, temperature_top=0.0)
    for flags in (0, capi.FLAG_INDEX_FROM_BOTTOM):
        out, st, rc = gpu_lib.flux_solve(w, flags)
        top = -1 if flags else 0
        assert rc == 0 and not st.any()
        check_top(out["flux_down"][:, top], out["mean_intensity_down"][:, top], incoming)
    _, st, jac, rc = gpu_lib.flux_solve_jac(w)
    assert rc == 0 and not st.any()
    assert not jac["flux_down"][:, 0].any() and not jac["mean_intensity_down"][:, 0].any()


@pytest.mark.parametrize("incoming", [0.0, 0.3])
@pytest.mark.parametrize("beam", [False, True])
@pytest.mark.parametrize("N", [4, 6, 8, 14, 16, 32, 64])
def test_general_path(N, beam, incoming):
    rng = np.random.default_rng(N)
    insts = []
    for k in range(3):
        L = (1, 6, 19)[k]
        dtau = np.clip(rng.lognormal(-1.0, 1.5, L), 1e-4, 10.0)
        insts.append(dict(num_streams=N, num_layers=L, num_phase_func_moments=N + 1, delta_tau=dtau,
                          single_scat_albedo=rng.uniform(0.0, 0.99, L),
                          phase_function_moments=workloads.hg_moments(rng.uniform(0.3, 0.9, L), N + 2),
                          temperature=200.0 + 90.0 * rng.random(L + 1), wavenumber_low=500.0, wavenumber_high=510.0,
                          temperature_bottom=290.0, temperature_top=0.0, isotropic_flux_top=incoming,
                          direct_beam_flux=1.0 if beam else 0.0, direct_beam_mu=0.6, surface_albedo=0.3,
                          tau_user=[0.0, workloads.column_total(dtau)], mu_user=[-0.8, 0.4], phi_user=[0.0]))
    for flags in (capi.GFLAG_USER_TAU | capi.GFLAG_USER_MU, capi.GFLAG_ONLY_FLUXES):
        d = capi.pack_general(insts, flags | capi.FLAG_THERMAL)
        got, rc = gpu_lib.general_solve(d)
        assert rc == 0 and not got["status"].any()
        check_top(got["flux_down"][:, 0], got["mean_intensity_down"][:, 0], incoming, 0.6 if beam else 0.0)
        batch, keep = capi.make_general_batch(d)
        outs, o, keep2 = capi.alloc_general_out_numpy(d)
        jac, jo, keep3 = capi.alloc_general_jac_numpy(d)
        if N % 4 == 0:
            assert gpu_lib.context().general_bands_solve_jac(batch, o, jo) == 0
            assert not jac["flux_down"][:, 0].any() and not jac["mean_intensity_down"][:, 0].any()
