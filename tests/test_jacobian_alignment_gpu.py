"""GPU test of temperature Jacobians where half the stream count and the number of
degrees of freedom are both odd (6, 10, 14 streams, an odd number of layers): the
records behind the Jacobians' vectors are read with 16-byte copies and have to start on
a boundary whatever the vectors' size.  Parity as in test_jacobian_gpu.py; single
columns and ragged batches of an odd number of layers in all."""
import numpy as np
import pytest

from disort_b200 import capi, workloads
from test_jacobian_gpu import check, general_check, general_thermal_mix

pytestmark = pytest.mark.gpu


def column(N, L):
    inst = general_thermal_mix(1, seed=10 * N + L, nstr=(N,))[0]
    rng = np.random.default_rng(L)
    dtau = np.clip(rng.lognormal(-2.0, 1.5, L), 1e-4, 5.0)
    inst.update(num_layers=L, delta_tau=dtau, single_scat_albedo=rng.uniform(0.0, 0.95, L),
                phase_function_moments=workloads.hg_moments(rng.uniform(0.0, 0.9, L), N + 1),
                temperature=200.0 + 100.0 * rng.random(L + 1), tau_user=[0.0, 0.4 * workloads.column_total(dtau)])
    return inst


@pytest.mark.parametrize("flags", [capi.GFLAG_USER_TAU | capi.GFLAG_USER_MU, capi.GFLAG_ONLY_FLUXES])
@pytest.mark.parametrize("N", [6, 10, 14])
@pytest.mark.parametrize("layers", [(1,), (3,), (33,), (3, 5, 1), (8, 7, 4)])
def test_general_path(N, layers, flags):
    general_check([column(N, L) for L in layers], capi.FLAG_THERMAL | flags, f"N={N} layers={layers}")


@pytest.mark.parametrize("N", [6, 10, 14])
@pytest.mark.parametrize("n,L", [(1, 1), (3, 7), (5, 33)])
def test_flux_path(N, n, L):
    check(workloads.thermal_sweep(n_bands=n, num_layers=L, num_streams=N, seed=N + L), label=f"N={N} n={n} L={L}")
