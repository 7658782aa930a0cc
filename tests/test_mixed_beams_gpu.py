"""GPU test of thermal batches in which some columns have a beam and some have none.

Columns share a warp of the boundary-value kernel: one whose beam ends at the
absorption cut must not reach a neighbour that has no beam, whose layer records hold no
beam terms (whatever was in memory there).  Every column is compared bit for bit with
the same column solved in a batch where nobody has a beam, or where all have theirs.
To make what is left in memory visible, the scratch is filled with NaN before each
solve and a batch with an infinite beam is solved first, which leaves NaN and infinity
in the shared memory of every kernel; both forms of the layer stage.
"""
import numpy as np
import pytest

import gpu_lib
from disort_b200 import capi

pytestmark = pytest.mark.gpu


def columns(N, n, L, fbeam):
    rng = np.random.default_rng(N + n)
    moments = np.broadcast_to(0.5 ** np.arange(N + 1), (n, L, N + 1)).copy()
    lo = rng.uniform(300.0, 900.0, n)
    return dict(n_inst=n, num_streams=N, num_layers=L, num_phase_func_moments=0, pmom_count=N + 1,
                flags=capi.FLAG_THERMAL,
                arrays=dict(wavenumber_low=lo, wavenumber_high=lo + 5.0, delta_tau=rng.uniform(0.5, 4.0, (n, L)),
                            single_scat_albedo=rng.uniform(0.0, 0.6, (n, L)), phase_function_moments=moments,
                            temperature=200.0 + 90.0 * rng.random(L + 1), surface_albedo=rng.uniform(0.0, 0.5, n),
                            emissivity_top=1.0, direct_beam_flux=fbeam, direct_beam_mu=rng.uniform(0.2, 0.9, n),
                            isotropic_flux_top=0.0, isotropic_flux_bottom=0.0, temperature_top=0.0,
                            temperature_bottom=290.0))


@pytest.mark.parametrize("jacobian", [False, True])
@pytest.mark.parametrize("stage", [1, 2])
@pytest.mark.parametrize("N", [4, 6, 8, 10, 12, 14, 16])
def test_columns_without_a_beam_beside_columns_past_their_cut(N, stage, jacobian):
    n, L = 37, 12
    ctx = gpu_lib.context()
    beams = np.where(np.arange(n) % 3 == 0, 0.0, 1.5)

    def solve(fbeam):
        solver = gpu_lib.flux_solve_jac if jacobian else gpu_lib.flux_solve
        solver(columns(N, 600, L, np.full(600, np.inf)))
        out = solver(columns(N, n, L, fbeam))
        assert out[-1] == 0 and not out[1].any()
        return dict(out[0], **({"d" + k: v for k, v in out[2].items()} if jacobian else {}))

    assert ctx.set_schedule([(N, 1, 1000000, stage, 0, 0)]) == 0
    ctx.set_debug(capi.DEBUG_POISON_SCRATCH)
    try:
        mixed, none, lit = solve(beams), solve(np.zeros(n)), solve(np.full(n, 1.5))
    finally:
        ctx.set_debug(0)
        ctx.load_schedule_file(capi.TUNING_FILE)
    for f, v in mixed.items():
        assert np.isfinite(v).all(), f
        np.testing.assert_array_equal(v[beams == 0.0], none[f][beams == 0.0], err_msg=f)
        np.testing.assert_array_equal(v[beams > 0.0], lit[f][beams > 0.0], err_msg=f)
