"""GPU test of the pieces that a flux batch in host memory is cut into (dsp_capi.cu): a
column's result does not depend on the piece it falls into, so the outputs are the bits
of the device-memory solve, at sizes on both sides of each change of the number of
pieces (16 MB of inputs and outputs), with as many instances as a multiple of 64 and
one more, with Jacobians, and in a workspace that holds a fraction of the batch."""
import numpy as np
import pytest

import gpu_lib
from disort_b200 import capi, workloads

pytestmark = pytest.mark.gpu


def same(w, jacobian):
    if jacobian:
        host, hst, hj, rc = gpu_lib.flux_solve_jac(w)
        dev, dst, dj, rc2 = gpu_lib.flux_solve_jac_device(w)
        host, dev = dict(host, **{"d" + k: v for k, v in hj.items()}), dict(dev, **{"d" + k: v for k, v in dj.items()})
    else:
        host, hst, rc = gpu_lib.flux_solve(w)
        dev, dst, rc2 = gpu_lib.flux_solve_device(w)
    assert rc == 0 and rc2 == 0
    np.testing.assert_array_equal(hst, dst)
    for f in host:
        np.testing.assert_array_equal(host[f], dev[f], err_msg=f)


def bytes_per_column(w):
    a = w["arrays"]
    per = sum(v[0].nbytes if v.ndim > 1 else 8 for k, v in a.items()
              if isinstance(v, np.ndarray) and v.ndim and len(v) == w["n_inst"])
    return per + 8 * 8 * (w["num_layers"] + 1) + 4


@pytest.mark.parametrize("workspace", [None, "24"])
@pytest.mark.parametrize("pieces", [2, 3, 7])
@pytest.mark.parametrize("N,L", [(4, 40), (8, 23), (16, 60)])
def test_pieces(monkeypatch, N, L, pieces, workspace):
    if workspace:
        monkeypatch.setenv("DSP_WORKSPACE_MB", workspace)
    one = bytes_per_column(workloads.thermal_sweep(n_bands=8, num_layers=L, num_streams=N, seed=1))
    for n in (pieces * 16_000_000 // one - 1, (pieces * 16_000_000 // one + 65) // 64 * 64 + 1):
        w = workloads.thermal_sweep(n_bands=n, num_layers=L, num_streams=N, seed=n)
        w["arrays"].update(direct_beam_flux=np.where(np.arange(n) % 3, 1.0, 0.0), direct_beam_mu=0.4)
        same(w, False)


@pytest.mark.parametrize("N,L,n", [(4, 13, 1999), (6, 7, 5001), (16, 30, 777)])
def test_pieces_with_jacobians(N, L, n):
    same(workloads.thermal_sweep(n_bands=n, num_layers=L, num_streams=N, seed=n), True)
