"""FP64 operation counts of one DISORT solve (the roofline numerators), by kernel.

Counted is what the algorithm in use cannot do without, h = N/2, a multiplication and
an addition as two operations:

* layer stage: the two halves of the phase matrix 2 N h^2, two Cholesky factors and
  their product 5/3 h^3; the eigenvectors of the h x h product as a symmetric QR
  iteration would need them, 16.33 h^3 + 6 h^2 (the Jacobi sweeps take more), recovery
  of X and Y 2 h^3, particular solutions 8 h^2 each;
* boundary-value problem, modal form (csrc/flux_bvp.cuh): per layer two symmetric
  inverses 2 h^3 each and four h^3 products of 2 operations, 12 h^3 in all, or six
  (16 h^3) with transmission records (N <= 16, fluxes only), and its matrix-vector
  products, 24 h^2.  The band factorisation of the reference (FluxSolver.cpp:838-1131)
  needs about ten times as many; band_lu_flops counts those for comparison.
* general path, per azimuth mode: the same; the user angles 2 (N - m) h + 4 h^2 per
  layer and angle; intensities 8 N per layer, output depth and angle.

Transcendental calls (exp, sqrt, log, pow) are not counted.
"""
from __future__ import annotations

import functools


def front_flops(N: int, nact: int | None = None) -> float:
    """Phase sums and factors of one layer with nact active Legendre orders."""
    h = N / 2
    return 2.0 * (N if nact is None else nact) * h * h + 5.0 / 3.0 * h ** 3


def eigen_flops(N: int, sources: int) -> float:
    """Eigenvectors, X and Y, and the particular solutions of one layer."""
    h = N / 2
    return 18.33 * h ** 3 + 6 * h * h + sources * 8 * h * h


def modal_bvp_flops(N: int, lean: bool) -> float:
    """Both passes over one layer."""
    h = N / 2
    return (16.0 if lean else 12.0) * h ** 3 + 24 * h * h


@functools.lru_cache(maxsize=None)
def band_lu_flops(N: int, ncut: int) -> float:
    NN = N // 2
    ml = mu = 3 * NN - 1
    n = N * ncut
    fac = 0.0
    sol = 0.0
    for k in range(1, n):
        lm = min(ml, n - k)
        fac += 2.0 * lm * min(ml + mu, n - k)
        sol += 2.0 * lm
    m1 = ml + mu + 1
    for k in range(1, n + 1):
        sol += 2.0 * (min(k, m1) - 1)
    return fac + sol


def flux_solve_flops(N: int, L: int, beam: bool, thermal: bool, ncut: int | None = None) -> dict:
    """FLOPs of one flux solve split by the engine kernel that performs each part."""
    nc = L if ncut is None else ncut
    front, eigen = nc * front_flops(N), nc * eigen_flops(N, int(beam) + int(thermal))
    if N > 16:  # one kernel for the layer stage
        front, eigen = front + eigen, 0.0
    bvp = nc * modal_bvp_flops(N, N <= 16) + (L + 1) * 8.0 * N
    return {"flux_layer_kernel": front, "flux_eigen_kernel": eigen, "flux_bvp_kernel": bvp,
            "total": front + eigen + bvp}


def absorption_cut(dtau, ssa, thermal: bool) -> int:
    """Layers the solvers keep (disortSet's abscut = 10 absorption depth rule)."""
    L = len(dtau)
    abstau, ncut = 0.0, L
    for lc in range(L):
        if abstau < 10.0:
            ncut = lc + 1
        abstau += (1.0 - ssa[lc]) * dtau[lc]
    lyrcut = abstau >= 10.0 and not thermal and L > 1
    return ncut if lyrcut else L


def general_solve_flops(N: int, L: int, ncut: int, modes: int, numu: int, ntau: int, beam: bool,
                        thermal: bool) -> dict:
    """FLOPs of one general (DisortSolver) solve, split by engine kernel."""
    h = N / 2
    lay = angle = bvp = inten = 0.0
    for m in range(modes):
        nact = N - m
        lay += ncut * (front_flops(N, nact) + eigen_flops(N, int(beam) + int(thermal and m == 0)))
        angle += ncut * numu * (2.0 * nact * h + 4.0 * h * h)
        bvp += ncut * modal_bvp_flops(N, False)
        if m == 0:
            bvp += ntau * (8.0 * h * h + 8.0 * N)
        inten += 8.0 * N * ntau * numu * ncut
    return {"gen_layer_kernel": lay, "gen_angle_kernel": angle, "gen_bvp_kernel": bvp,
            "gen_intensity_kernel": inten, "total": lay + angle + bvp + inten}
