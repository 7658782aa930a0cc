"""GPU test of columns of layers with exactly one of -A_s and -B_s positive definite
(unphysical moments): the eigensolver's other branch, and matrices in the boundary-value
problem that are not positive definite (csrc/flux_layer.cuh, csrc/flux_bvp.cuh).  From a
moment just past definite to 60; thin and (up to 16 streams, where the oracle's two
builds still agree to 2e-11) thick layers; tasks of a warp mixed, all of one kind, and alone; both
parities of azimuth mode (general solver).  The result of a column does not depend on
its neighbours (bit for bit), and is the oracle's to 1e-9 and four times what the
oracle's two builds differ by (such columns amplify rounding), as in
test_modal_bvp_gpu.py."""
import numpy as np
import pytest

import gpu_lib
import oracle_lib
from disort_b200 import capi
from test_modal_bvp_gpu import columns

pytestmark = pytest.mark.gpu


def moments(N, n, L, which, seed, thick=False):
    """Even columns get, in every layer, an even (0) or odd (1) moment from 1 to 60."""
    rng = np.random.default_rng(seed)
    w = columns(N, n, L, seed, True, ssa=0.9)
    w["arrays"]["delta_tau"] = np.clip(w["arrays"]["delta_tau"], 0.01, 0.3) * (100.0 if thick else 1.0)
    pm = w["arrays"]["phase_function_moments"]
    pm[:, :, 1:] *= 0.2
    pm[::2, :, 2 if which == 0 else 1] = np.geomspace(1.0, 60.0, (n + 1) // 2)[:, None] * rng.uniform(0.9, 1.1)
    pm[:, :, N] = 0.0
    return w


def part(w, keep):
    a = {k: v[keep] if isinstance(v, np.ndarray) and v.ndim and len(v) == w["n_inst"] and k != "temperature" else v
         for k, v in w["arrays"].items()}
    return dict(w, n_inst=len(keep), arrays=a)


@pytest.mark.parametrize("N,thick", [(n, False) for n in capi.SUPPORTED_NSTR] + [(n, True) for n in (4, 6, 8, 10, 12, 14, 16)])
@pytest.mark.parametrize("which", [0, 1])
def test_mixed_and_alone(N, which, thick):
    w = moments(N, 39, 3, which, 5 * N + which, thick)
    got, gst, rc = gpu_lib.flux_solve(w)
    assert rc == 0
    for keep in (np.arange(0, 39, 2), np.arange(1, 39, 2), np.array([0]), np.array([38])):
        sub, sst, rc = gpu_lib.flux_solve(part(w, keep))
        assert rc == 0
        np.testing.assert_array_equal(sst, gst[keep])
        for f in got:
            np.testing.assert_array_equal(sub[f], got[f][keep], err_msg=f)
    ref, rst = oracle_lib.flux_solve(w, ext=True)
    dbl, _ = oracle_lib.flux_solve(w)
    np.testing.assert_array_equal(gst, rst)
    ok = gst == 0
    assert ok[1::2].all() and ok[::2].sum() >= 5
    for f in got:
        spread = np.max(np.abs(dbl[f] - ref[f]) / (np.abs(ref[f]) + 1e-3), axis=1, where=ok[:, None], initial=0.0)[:, None]
        off = np.abs(got[f] - ref[f])
        assert (off <= (1e-9 + 4.0 * spread) * np.abs(ref[f]) + 1e-12 + 4e-3 * spread)[ok].all(), f


@pytest.mark.parametrize("N,thick", [(n, False) for n in (4, 8, 16, 32)] + [(n, True) for n in (4, 8, 16)])
@pytest.mark.parametrize("which", [0, 1])
def test_azimuth_modes(N, which, thick):
    w = moments(N, 9, 2, which, 3 * N + which, thick)
    a = w["arrays"]
    insts = [dict(num_streams=N, num_layers=2, num_phase_func_moments=N, delta_tau=a["delta_tau"][k],
                  single_scat_albedo=a["single_scat_albedo"][k], phase_function_moments=a["phase_function_moments"][k],
                  direct_beam_flux=1.0, direct_beam_mu=0.6, surface_albedo=0.2,
                  tau_user=[0.0, float(a["delta_tau"][k].sum()) / 2.0], mu_user=[-0.7, 0.3], phi_user=[0.0, 50.0])
             for k in range(9)]
    d = capi.pack_general(insts, capi.GFLAG_USER_TAU | capi.GFLAG_USER_MU)
    got, rc = gpu_lib.general_solve(d)
    ref, dbl = oracle_lib.general_solve(d, ext=True), oracle_lib.general_solve(d)
    assert rc == 0
    np.testing.assert_array_equal(got["status"], ref["status"])
    ok = got["status"] == 0
    assert ok[1::2].all() and ok[::2].any()
    for f in ref:
        if f == "status":
            continue
        flat = lambda v: v[ok].reshape(int(ok.sum()), -1)  # noqa: E731
        g, r, b = flat(got[f]), flat(ref[f]), flat(dbl[f])
        size = np.maximum(np.abs(r), np.abs(r).max(1, keepdims=True) if f.startswith("int") else 0.0)
        spread = np.max(np.abs(b - r) / (size + 1e-3), axis=1, keepdims=True)
        assert (np.abs(g - r) <= (1e-9 + 4.0 * spread) * size + 1e-12 + 4e-3 * spread).all(), f


@pytest.mark.parametrize("N,thick", [(4, False), (4, True), (6, True), (16, False), (16, True), (32, False)])
@pytest.mark.parametrize("which", [0, 1])
def test_jacobians(N, thick, which):
    """Temperature derivatives of such columns, held as in test_jacobian_gpu.py."""
    from test_jacobian_gpu import jac_ratio
    w = moments(N, 9, 3, which, 2 * N + which, thick)
    out, st, jac, rc = gpu_lib.flux_solve_jac(w)
    rout, rst, rjac = oracle_lib.flux_solve_jac(w, ext=True)
    assert rc == 0 and not st.any() and not rst.any()
    r, where = jac_ratio(jac, rjac)
    assert r <= 1.0, where
