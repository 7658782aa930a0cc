"""GPU test of the layer eigensolver where two columns of the one-sided Jacobi
iteration have equal norms, so that the rotation is by 45 degrees.

At 4 streams there is one pair of columns, F = L^T R of the factors of -B_s and -A_s
(csrc/flux_layer.cuh): a rotation left out leaves the layer's modes wrong.  Columns of
one layer whose omega makes the norms equal (by bisection, for random moments), or
equal to some parts in 1e5 to 1e9.  Checker: the extended-precision oracle, by the
parity of tests/parity.py.
"""
import numpy as np
import pytest

import gpu_lib
import oracle_lib
from disort_b200 import capi
from parity import assert_parity

pytestmark = pytest.mark.gpu


def column_norms(ssa, pm):
    """Squared norms of the two columns of F for 4 streams (NaN where a matrix is indefinite)."""
    mu = np.array([0.5 * (1.0 + 1.0 / np.sqrt(3.0)), 0.5 * (1.0 - 1.0 / np.sqrt(3.0))])  # the solver's order
    d = np.sqrt(0.5 * mu)
    P = np.array([np.ones(2), mu, 0.5 * (3 * mu ** 2 - 1), 0.5 * (5 * mu ** 3 - 3 * mu)])
    g = (2 * np.arange(4) + 1) * ssa[:, None] * pm
    factors = []
    for ls in ((1, 3), (0, 2)):
        S = sum(g[:, l, None, None] * np.outer(P[l], P[l]) for l in ls)
        M = d[:, None] * (np.eye(2) - 0.5 * S) / mu[:, None] / d
        a = np.sqrt(M[:, 0, 0])
        b = M[:, 1, 0] / a
        factors.append((a, b, np.sqrt(M[:, 1, 1] - b * b)))
    (l0, l1, l2), (r0, r1, r2) = factors
    return (l0 * r0 + l1 * r1) ** 2 + (l2 * r1) ** 2, (l1 * r2) ** 2 + (l2 * r2) ** 2


def equal_norm_columns(n, seed):
    """(omega, moments) of n layers whose columns have equal norms."""
    rng = np.random.default_rng(seed)
    pm = np.concatenate([np.ones((8 * n, 1)), rng.uniform(-1.0, 1.0, (8 * n, 3))], axis=1)
    lo, hi = np.full(8 * n, 0.05), np.full(8 * n, 0.98)
    a, b = column_norms(lo, pm)
    c, d = column_norms(hi, pm)
    use = np.flatnonzero((a < b) & (c > d))[:n]
    pm, lo, hi = pm[use], lo[use], hi[use]
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        a, b = column_norms(mid, pm)
        lo, hi = np.where(a < b, mid, lo), np.where(a < b, hi, mid)
    return 0.5 * (lo + hi), pm


@pytest.mark.parametrize("stage", [1, 2])
def test_columns_of_equal_norm(stage):
    n = 1200
    ssa, pm = equal_norm_columns(n, 3)
    assert len(ssa) == n
    ssa *= 1.0 + np.where(np.arange(n) % 2, 10.0 ** np.linspace(-9.0, -5.0, n), 0.0)
    pc = 5
    moments = np.zeros((n, 1, pc))  # (no delta-M)
    moments[:, 0, :4] = pm
    w = dict(n_inst=n, num_streams=4, num_layers=1, num_phase_func_moments=0, pmom_count=pc, flags=capi.FLAG_THERMAL,
             arrays=dict(wavenumber_low=500.0 * np.ones(n), wavenumber_high=505.0 * np.ones(n),
                         delta_tau=np.full((n, 1), 0.3), single_scat_albedo=ssa[:, None],
                         phase_function_moments=moments, temperature=np.array([220.0, 280.0]),
                         surface_albedo=0.2 * np.ones(n), emissivity_top=1.0, direct_beam_flux=2.0,
                         direct_beam_mu=0.63 * np.ones(n), isotropic_flux_top=0.1, isotropic_flux_bottom=0.0,
                         temperature_top=150.0, temperature_bottom=290.0))
    ctx = gpu_lib.context()
    assert ctx.set_schedule([(4, 1, 1000000, stage, 0, 0)]) == 0
    try:
        got, gst, rc = gpu_lib.flux_solve(w)
    finally:
        ctx.load_schedule_file(capi.TUNING_FILE)
    ref, rst = oracle_lib.flux_solve(w, ext=True)
    assert rc == 0 and not gst.any() and not rst.any()
    assert_parity(got, ref, f"layer stage {stage}")
