"""The solves that performance is measured on, each through a public entry point.

listed()  the named cases: single columns through the solver objects, spectral loops of
          every stream-count class in device and host memory, temperature Jacobians, the
          general solver's radiances, and the flux emulator's training step and inference.
draw()    further cases of the same ranges.
prepare() the inputs and handles a program holds before the call, run() one call,
exact()   the same results in plain 64-bit torch: eigenvectors of each layer, the
          reflection of the column above carried down, radiances by analytic integration.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import disort_b200 as db
from disort_b200 import capi

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
STREAMS = (4, 6, 8, 10, 12, 14, 16, 32, 64)


def _flux(name, n, layers, streams, thermal=True, beam=False, dmplus=False, bottom_up=False, memory="device",
          hg=False, jacobian=False):
    return dict(name=name, kind="flux", n=n, layers=layers, streams=streams, thermal=thermal, beam=beam,
                dmplus=dmplus, bottom_up=bottom_up, memory=memory, hg=hg, jacobian=jacobian)


def _general(name, n, streams, lmin, lmax, beam=True, thermal=False, dmplus=True, ntau=3, numu=5, nphi=4,
             memory="device"):
    return dict(name=name, kind="general", n=n, streams=streams, lmin=lmin, lmax=lmax, beam=beam, thermal=thermal,
                dmplus=dmplus, ntau=ntau, numu=numu, nphi=nphi, memory=memory)


def listed():
    return [
        # one column and one band through a solver object: what an interactive user or a
        # column model that calls band by band waits for
        dict(name="column_16str", kind="column", layers=60, streams=16),
        # the 1,024-band solar sweep over a shallow column from Python arrays
        dict(name="bands_beam_16str", kind="bands", n=1024, layers=4, streams=16),
        # the line-by-line thermal sweep of bench.py, inputs resident on the GPU
        _flux("sweep_thermal_16str", 20000, 60, 16),
        # a spectral loop fed from pinned host memory with one asymmetry factor per layer,
        # thermal and solar, bottom-up arrays as climate models keep them
        _flux("sweep_host_8str", 8191, 47, 8, beam=True, bottom_up=True, memory="host", hg=True),
        # the cheap 4-stream solve of very many columns (the emulator's first step)
        _flux("columns_4str", 60000, 40, 4, beam=True),
        # high-accuracy fluxes of deep columns with forward-peaked scattering
        _flux("deep_64str", 192, 91, 64, beam=True, dmplus=True),
        # fluxes with their temperature Jacobians, the linearisation a retrieval takes
        _flux("jacobians_16str", 256, 50, 16, jacobian=True),
        # the general solver's ragged mix: 4 to 64 streams, 10 to 120 layers, every azimuth mode
        _general("radiance_mix", 1024, 0, 10, 120),
        # radiances of one stream count from host memory, the usual satellite simulation
        _general("radiance_16str_host", 1000, 16, 10, 120, memory="host"),
        # one column's radiances through the general solver object
        dict(name="radiance_32str", kind="radiance", layers=33, streams=32),
        # the flux emulator: forward and backward of one training batch, and inference
        dict(name="emulator_gradients", kind="emulator", rows=4096, training=True),
        dict(name="emulator_forward", kind="emulator", rows=65536, training=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.5:
        N = rng.choice(STREAMS)
        L = _log_int(rng, 3, 130)
        # layers in all, so that deep or many-stream columns come in smaller batches
        cap = {4: 3e6, 6: 2e6, 8: 2e6, 10: 1.5e6, 12: 1.2e6, 14: 1.2e6, 16: 1.2e6, 32: 1.2e5, 64: 1.8e4}[N]
        c = _flux("", _log_int(rng, 2, max(3, min(60000, int(cap / L)))), L, N)
        c["beam"] = rng.random() < 0.5
        c["thermal"] = not c["beam"] or rng.random() < 0.7
        c["dmplus"] = rng.random() < 0.3
        c["bottom_up"] = rng.random() < 0.2
        c["memory"] = "host" if rng.random() < 0.35 else "device"
        c["hg"] = rng.random() < 0.3
        if c["thermal"] and rng.random() < 0.15:
            c["jacobian"] = True
            c["n"] = max(2, min(c["n"], int(20000 * 16 / (L * N)), int(4e6 / (L * L))))
    elif pick < 0.85:
        N = rng.choice((0,) + STREAMS)
        lmin = _log_int(rng, 2, 40)
        lmax = lmin + rng.randint(0, 80)
        mean = 0.5 * (lmin + lmax)
        cap = {0: 4e4, 4: 1.5e6, 6: 8e5, 8: 5e5, 10: 3e5, 12: 2e5, 14: 1.5e5, 16: 1e5, 32: 3e4, 64: 3e3}[N]
        c = _general("", _log_int(rng, 2, max(3, min(4000, int(cap / mean)))), N, lmin, lmax)
        c["thermal"] = rng.random() < 0.3
        c["beam"] = not c["thermal"] or rng.random() < 0.7
        c["dmplus"] = rng.random() < 0.6
        c["ntau"], c["numu"], c["nphi"] = rng.randint(1, 6), rng.randint(1, 12), rng.randint(1, 6)
        c["memory"] = "host" if rng.random() < 0.4 else "device"
    elif pick < 0.90:
        c = dict(kind="column", layers=_log_int(rng, 3, 130), streams=rng.choice(STREAMS))
    elif pick < 0.95:
        c = dict(kind="bands", n=_log_int(rng, 8, 4000), layers=_log_int(rng, 2, 40), streams=rng.choice(STREAMS[:7]))
    else:
        c = dict(kind="emulator", rows=128 * _log_int(rng, 4, 400), training=rng.random() < 0.4)
        if c["training"]:
            c["rows"] = min(c["rows"], 8192)
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# inputs (numpy, from the seed alone)
# ---------------------------------------------------------------------------
def _levels(rng, L):
    return 180.0 + 140.0 * np.arange(L + 1) / L + rng.uniform(-10.0, 10.0, L + 1)


def _flux_inputs(c, seed):
    """Atmospheric columns as workloads.thermal_sweep draws them, with the case's options."""
    rng = np.random.default_rng(seed)
    n, L, N = c["n"], c["layers"], c["streams"]
    wide = min(0.14 * 20000 / n, 25.0)
    lo = 100.0 + wide * np.arange(n) % 2800.0
    d = dict(lo=lo, hi=lo + wide, dtau=np.clip(rng.lognormal(-3.0, 2.0, (n, L)), 1e-6, 50.0),
             ssa=rng.uniform(0.0, 0.99, (n, L)),
             g=rng.uniform(0.5, 0.95, (n, L)) if c["dmplus"] else rng.uniform(0.0, 0.9, (n, L)),
             temp=_levels(rng, L), albedo=rng.uniform(0.0, 0.6, n), mu0=rng.uniform(0.1, 0.99, n))
    d["fbeam"] = 1.0 if c["beam"] else 0.0
    d["nmom"] = N + 1 if c["dmplus"] else 0
    if c["bottom_up"]:
        d["temp"] = d["temp"][::-1].copy()
    return d


MU5 = (-0.5, -0.1, 0.1, 0.5, 1.0)
PHI4 = (0.0, 60.0, 120.0, 180.0)


def _angles(c):
    if c["numu"] == 5:
        mu = MU5
    else:
        neg = np.linspace(-0.97, -0.12, c["numu"] // 2)
        pos = np.linspace(0.07, 0.93, c["numu"] - c["numu"] // 2)
        mu = np.concatenate([neg, pos])
    phi = PHI4 if c["nphi"] == 4 else np.linspace(0.0, 175.0, c["nphi"])
    return np.asarray(mu, dtype=np.float64), np.asarray(phi, dtype=np.float64)


def _column_total(dtau):
    return min(np.add.accumulate(dtau)[-1], np.add.accumulate(dtau[::-1])[-1])


def _general_inputs(c, seed):
    """A ragged batch as workloads.general_mix draws it, in the layout of pack_general."""
    rng = np.random.default_rng(seed)
    n = c["n"]
    if c["streams"]:
        N = np.full(n, c["streams"], dtype=np.int32)
    else:
        N = rng.choice(np.array([4, 8, 16, 32, 64], dtype=np.int32), size=n, p=[0.1, 0.2, 0.4, 0.2, 0.1])
    L = rng.integers(c["lmin"], c["lmax"] + 1, n).astype(np.int32)
    off = np.zeros(n + 1, dtype=np.int64)
    off[1:] = np.cumsum(L)
    tot = int(off[-1])
    pc = int(N.max()) + 2
    dtau = np.clip(rng.lognormal(-3.0, 2.0, tot), 1e-6, 50.0)
    g = rng.uniform(0.5, 0.95, tot)
    temp = 180.0 + 140.0 * np.concatenate([np.arange(k + 1) / k for k in L]) + rng.uniform(-10.0, 10.0, tot + n)
    total = np.array([_column_total(dtau[off[i]:off[i + 1]]) for i in range(n)])
    frac = np.linspace(0.0, 1.0, c["ntau"]) if c["ntau"] > 1 else np.array([0.5])
    mu, phi = _angles(c)
    flags = capi.GFLAG_USER_TAU | capi.GFLAG_USER_MU
    flags |= capi.FLAG_DELTA_M_PLUS if c["dmplus"] else 0
    flags |= capi.FLAG_THERMAL if c["thermal"] else 0
    one = np.ones(n)
    return dict(n_inst=n, flags=flags, num_streams=N, num_layers=L, layer_offset=off,
                num_phase_func_moments=(N + 1).astype(np.int32), pmom_count=pc, accuracy=0.0, delta_tau=dtau,
                single_scat_albedo=rng.uniform(0.0, 0.99, tot),
                phase_function_moments=g[:, None] ** np.arange(pc, dtype=np.float64)[None, :], temperature=temp,
                tau_user=(np.minimum(total[:, None] * frac[None, :], total[:, None]), c["ntau"]), mu_user=(mu, 0),
                phi_user=(phi, 0), num_user_tau=c["ntau"], num_user_mu=len(mu), num_phi=len(phi), brdf_type=0,
                ntau_out=c["ntau"], numu_out=len(mu), wavenumber_low=600.0 * one, wavenumber_high=601.5 * one,
                surface_albedo=rng.uniform(0.0, 0.6, n), emissivity_top=one,
                direct_beam_flux=one * (1.0 if c["beam"] else 0.0), direct_beam_mu=rng.uniform(0.1, 0.99, n),
                direct_beam_phi=0.0 * one, isotropic_flux_top=0.0 * one, isotropic_flux_bottom=0.0 * one,
                temperature_top=0.0 * one, temperature_bottom=temp[off[1:] + np.arange(n)])


def _one_column(c, seed):
    rng = np.random.default_rng(seed)
    L = c["layers"]
    temp = _levels(rng, L)
    return dict(dtau=np.clip(rng.lognormal(-3.0, 2.0, L), 1e-6, 50.0), ssa=rng.uniform(0.0, 0.99, L),
                g=rng.uniform(0.5, 0.9, L), temp=temp, albedo=float(rng.uniform(0.0, 0.6)),
                mu0=float(rng.uniform(0.1, 0.99)))


def _bands_inputs(c, seed):
    rng = np.random.default_rng(seed)
    n, L = c["n"], c["layers"]
    lo = 100.0 + 10.0 * np.arange(n)
    return dict(lo=lo, hi=lo + 10.0, dtau=rng.uniform(0.01, 1.0, L) * rng.lognormal(0.0, 1.0, (n, 1)),
                ssa=rng.uniform(0.3, 0.999, (n, L)), g=0.8, albedo=rng.uniform(0.0, 0.3, n), mu0=0.5)


EMU = dict(n_in=658, hidden=512, n_hidden_layers=4, n_out=82, n_heads=2)


def _pad64(x):
    return (x + 63) // 64 * 64


def _emulator_dims():
    widths = [EMU["n_in"]] + [EMU["hidden"]] * EMU["n_hidden_layers"] + [EMU["n_out"] * EMU["n_heads"]]
    return list(zip(widths[:-1], widths[1:]))


def _emulator_inputs(c, seed):
    """Parameters [(W, b)] without padding, features, targets and head weights."""
    rng = np.random.default_rng(seed)
    params = [(rng.standard_normal((o, i)).astype(np.float32) * np.float32(math.sqrt(2.0 / i)),
               0.05 * rng.standard_normal(o).astype(np.float32)) for i, o in _emulator_dims()]
    x = rng.standard_normal((c["rows"], EMU["n_in"]), dtype=np.float32)
    y = rng.standard_normal((c["rows"], EMU["n_out"]), dtype=np.float32)
    hw = rng.poisson(1.0, (c["rows"], EMU["n_heads"])).astype(np.float32)
    return params, x, y, hw


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
_CONTEXT = None


def _context():
    """One engine context per program, as a user keeps it."""
    global _CONTEXT
    if _CONTEXT is None:
        _CONTEXT = capi.Context(0)
    return _CONTEXT


def _dev(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")


def _moments(g, count, device):
    """Henyey-Greenstein moments g**k by successive products."""
    g = torch.as_tensor(np.ascontiguousarray(g), device=device)
    m = torch.empty(g.shape + (count,), dtype=torch.float64, device=device)
    m[..., 0] = 1.0
    for k in range(1, count):
        m[..., k] = m[..., k - 1] * g
    return m


def _prepare_flux(c, seed):
    d = _flux_inputs(c, seed)
    n, L, N = c["n"], c["layers"], c["streams"]
    host = c["memory"] == "host"
    pc = max(N, d["nmom"]) + 1
    flags = ((capi.FLAG_THERMAL if c["thermal"] else 0) | (capi.FLAG_DELTA_M_PLUS if c["dmplus"] else 0) |
             (capi.FLAG_INDEX_FROM_BOTTOM if c["bottom_up"] else 0) | (capi.FLAG_HG_G if c["hg"] else 0) |
             (0 if host else capi.FLAG_DEVICE_POINTERS))
    put = (lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64)).pin_memory()) if host else _dev
    pm = put(d["g"]) if c["hg"] else _moments(d["g"], pc, "cuda")
    if host and not c["hg"]:
        pm = pm.cpu().pin_memory()
    one = lambda v: put(np.array([float(v)]))  # noqa: E731
    surface = d["temp"][0 if c["bottom_up"] else -1]
    arrays = dict(wavenumber_low=put(d["lo"]), wavenumber_high=put(d["hi"]), delta_tau=put(d["dtau"]),
                  single_scat_albedo=put(d["ssa"]), phase_function_moments=pm, temperature=put(d["temp"]),
                  surface_albedo=put(d["albedo"]), emissivity_top=one(1.0), direct_beam_flux=one(d["fbeam"]),
                  direct_beam_mu=put(d["mu0"]), isotropic_flux_top=one(0.0), isotropic_flux_bottom=one(0.0),
                  temperature_top=one(0.0), temperature_bottom=one(surface))
    where = dict(device="cpu", pin_memory=True) if host else dict(device="cuda")
    outs = {f: torch.zeros((n, L + 1), dtype=torch.float64, **where) for f in capi.FLUX_OUT_FIELDS}
    status = torch.zeros((n,), dtype=torch.int32, **where)
    batch, keep = capi.make_flux_batch(n, N, L, d["nmom"], pc, flags, arrays)
    out, keep2 = capi.make_flux_out(outs, status)
    s = dict(case=c, batch=batch, out=out, outs=outs, status=status, keep=(arrays, keep, keep2))
    if c["jacobian"]:
        s["jac"] = {f: torch.zeros((n, L + 1, L + 2), dtype=torch.float64, **where) for f in capi.JAC_FIELDS}
        s["jout"], s["keep3"] = capi.make_flux_jac_out(s["jac"])
    return s


def _prepare_general(c, seed):
    import ctypes
    d = _general_inputs(c, seed)
    host = c["memory"] == "host"
    if host:
        put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory()  # noqa: E731
    else:
        put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        d["flags"] |= capi.FLAG_DEVICE_POINTERS
    for k, v in list(d.items()):
        if isinstance(v, np.ndarray):
            d[k] = put(v)
        elif isinstance(v, tuple):
            d[k] = (put(v[0]), v[1])
    batch, keep = capi.make_general_batch(d)
    n, nt, nu, nphi = c["n"], c["ntau"], d["num_user_mu"], d["num_phi"]
    where = dict(device="cpu", pin_memory=True) if host else dict(device="cuda")
    outs = {f: torch.zeros((n, nt), dtype=torch.float64, **where) for f in capi.FLUX_OUT_FIELDS}
    outs["intensity"] = torch.zeros((n, nt, nu, nphi), dtype=torch.float64, **where)
    outs["intensity_azimuth_avg"] = torch.zeros((n, nt, nu), dtype=torch.float64, **where)
    status = torch.zeros((n,), dtype=torch.int32, **where)
    dp = lambda t: ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_double))  # noqa: E731
    o = capi.GeneralOut()
    for k, f in enumerate(capi.FLUX_OUT_FIELDS):
        o.flux[k] = dp(outs[f])
    o.intensity, o.intensity_azimuth_avg = dp(outs["intensity"]), dp(outs["intensity_azimuth_avg"])
    o.status = ctypes.cast(ctypes.c_void_p(status.data_ptr()), ctypes.POINTER(ctypes.c_int32))
    o.ntau_out, o.numu_out = nt, nu
    return dict(case=c, batch=batch, out=o, outs=outs, status=status, keep=(d, keep))


def _prepare_column(c, seed):
    d = _one_column(c, seed)
    cfg = db.DisortFluxConfig(c["layers"], c["streams"])
    cfg.use_thermal_emission = True
    cfg.wavenumber_low, cfg.wavenumber_high = 600.0, 610.0
    cfg.direct_beam_flux, cfg.direct_beam_mu, cfg.surface_albedo = 1.0, d["mu0"], d["albedo"]
    cfg.temperature_top, cfg.temperature_bottom = 0.0, float(d["temp"][-1])
    cfg.allocate()
    cfg.delta_tau, cfg.single_scat_albedo, cfg.temperature = d["dtau"].tolist(), d["ssa"].tolist(), d["temp"].tolist()
    cfg.phase_function_moments = _moments(d["g"], c["streams"] + 1, "cpu").tolist()
    return dict(case=c, config=cfg, solver=db.create_flux_solver(c["streams"]))


def _prepare_radiance(c, seed):
    d = _one_column(c, seed)
    cfg = db.DisortConfig(c["layers"], c["streams"], c["streams"] + 1)
    f = cfg.flags
    f.use_user_tau, f.use_user_mu, f.comp_only_fluxes = True, True, False
    f.use_thermal_emission, f.use_delta_m_plus = True, True
    cfg.wavenumber_low, cfg.wavenumber_high = 600.0, 610.0
    cfg.bc.direct_beam_flux, cfg.bc.direct_beam_mu, cfg.bc.direct_beam_phi = 1.0, d["mu0"], 0.0
    cfg.bc.surface_albedo, cfg.bc.temperature_top = d["albedo"], 0.0
    cfg.bc.temperature_bottom = float(d["temp"][-1])
    cfg.num_user_tau, cfg.num_user_mu, cfg.num_phi = 3, len(MU5), len(PHI4)
    cfg.allocate()
    cfg.delta_tau, cfg.single_scat_albedo, cfg.temperature = d["dtau"].tolist(), d["ssa"].tolist(), d["temp"].tolist()
    cfg.phase_function_moments = _moments(d["g"], c["streams"] + 2, "cpu").tolist()
    total = _column_total(d["dtau"])
    cfg.tau_user, cfg.mu_user, cfg.phi_user = [0.0, total / 2.0, total], list(MU5), list(PHI4)
    return dict(case=c, config=cfg, solver=db.DisortSolver())


def _prepare_bands(c, seed):
    d = _bands_inputs(c, seed)
    cfg = db.DisortFluxConfig(c["layers"], c["streams"])
    cfg.direct_beam_flux, cfg.direct_beam_mu, cfg.surface_albedo = math.pi, d["mu0"], 0.1
    cfg.allocate()
    cfg.set_henyey_greenstein(d["g"])
    return dict(case=c, config=cfg, bands=np.stack([d["lo"], d["hi"]], axis=1), d=d)


def _prepare_emulator(c, seed):
    from disort_b200.emu import Emulator
    params, x, y, hw = _emulator_inputs(c, seed)
    batch = c["rows"] if c["training"] else 4096
    emu = Emulator(batch=batch, seed=1, **EMU)
    flat = []
    for W, b in params:
        o, i = W.shape
        full = np.zeros((_pad64(o), _pad64(i)), dtype=np.float32)
        full[:o, :i] = W
        bias = np.zeros(_pad64(o), dtype=np.float32)
        bias[:o] = b
        flat += [full.ravel(), bias]
    emu.set_params(np.ascontiguousarray(np.concatenate(flat)))
    X = torch.zeros((c["rows"], emu.in_stride), dtype=torch.bfloat16, device="cuda")
    X[:, :EMU["n_in"]] = torch.from_numpy(x).cuda().to(torch.bfloat16)
    s = dict(case=c, emu=emu, X=X)
    if c["training"]:
        emu.set_data(X, torch.from_numpy(y).cuda(), torch.from_numpy(hw).cuda())
        s["grads"] = torch.zeros(emu.param_count(), dtype=torch.float32, device="cuda")
        s["loss"] = torch.zeros(1, dtype=torch.float32, device="cuda")
    else:
        s["preds"] = torch.zeros((c["rows"], EMU["n_out"] * EMU["n_heads"]), dtype=torch.float32, device="cuda")
    return s


def prepare(case, seed):
    return {"flux": _prepare_flux, "general": _prepare_general, "column": _prepare_column,
            "radiance": _prepare_radiance, "bands": _prepare_bands, "emulator": _prepare_emulator}[case["kind"]](
                case, seed)


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind in ("flux", "general"):
        ctx = _context()
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        if kind == "general":
            rc = ctx.general_bands_solve(s["batch"], s["out"])
        elif c["jacobian"]:
            rc = ctx.flux_bands_solve_jac(s["batch"], s["out"], s["jout"])
        else:
            rc = ctx.flux_bands_solve(s["batch"], s["out"])
        if rc != 0:
            raise RuntimeError(ctx.last_error())
        r = dict(s["outs"], status=s["status"])
        if c.get("jacobian"):
            r["jacobians"] = s["jac"]
        return r
    if kind == "column":
        res = s["solver"].solve(s["config"])
        return {f: np.asarray(getattr(res, f)) for f in capi.FLUX_OUT_FIELDS}
    if kind == "radiance":
        res = s["solver"].solve(s["config"])
        r = {f: np.asarray(getattr(res, f)) for f in capi.FLUX_OUT_FIELDS}
        r["intensity"] = np.asarray(res.intensity).reshape(-1)
        r["intensity_azimuth_avg"] = np.asarray(res.intensity_azimuth_avg).reshape(-1)
        return r
    if kind == "bands":
        d = s["d"]
        return db.solve_flux_spectral_bands_arrays(s["config"], s["bands"], delta_tau=d["dtau"],
                                                   single_scat_albedo=d["ssa"], surface_albedo=d["albedo"])
    if c["training"]:
        s["emu"].gradients(s["grads"], s["loss"])
        return dict(gradients=s["grads"], loss=s["loss"])
    s["emu"].forward(s["X"], s["preds"])
    return s["preds"]


# ---------------------------------------------------------------------------
# work: inputs read once, outputs written once; operations of the discrete-ordinate
# method with N/2 x N/2 matrices: per layer and azimuth mode the phase sums, a symmetric
# eigenproblem with vectors, its particular solutions, and the reflection of the layers
# above carried through the layer
# ---------------------------------------------------------------------------
def _layer_flops(N):
    h = N // 2
    return 2.0 * h * h * N + 9.0 * h ** 3 + 8.0 * h ** 3 + 12.0 * h * h


def work(case):
    c = case
    if c["kind"] == "emulator":
        p = sum(i * o for i, o in _emulator_dims())
        rows = c["rows"]
        return dict(flops=(6.0 if c["training"] else 2.0) * rows * p,
                    bytes=rows * (2.0 * EMU["n_in"] + 4.0 * EMU["n_out"] * (1 if c["training"] else 2)) +
                    (2.0 + (4.0 if c["training"] else 0.0)) * p)
    if c["kind"] == "general":
        Ns = [c["streams"]] if c["streams"] else [4, 8, 16, 32, 64]
        ws = [1.0] if c["streams"] else [0.1, 0.2, 0.4, 0.2, 0.1]
        L = 0.5 * (c["lmin"] + c["lmax"])
        pc = max(Ns) + 2
        per = sum(w * (N if c["beam"] else 1) * (_layer_flops(N) + 4.0 * c["numu"] * N * N) for w, N in zip(ws, Ns))
        return dict(flops=c["n"] * L * per,
                    bytes=8.0 * c["n"] * (L * (2 + pc) + c["ntau"] * (8 + c["numu"] * (1 + c["nphi"]))))
    n, L, N = c.get("n", 1), c["layers"], c["streams"]
    flops = n * L * _layer_flops(N)
    if c["kind"] == "radiance":
        return dict(flops=flops * N, bytes=8.0 * (L * (N + 4) + 3 * (8 + 25)))
    bytes_ = 8.0 * n * (L * (3 if c.get("hg") else 2 if c["kind"] == "bands" else N + 3) + 8 * (L + 1))
    if c.get("jacobian"):
        flops += n * L * (L + 2) * 8.0 * N * N
        bytes_ += 8.0 * 6 * n * (L + 1) * (L + 2)
    return dict(flops=flops, bytes=bytes_)


# ---------------------------------------------------------------------------
# exact: plain 64-bit torch
# ---------------------------------------------------------------------------
def _planck(lo, hi, T):
    """Band-integrated Planck radiance by the solver's own quadrature and series."""
    lo, hi, T = np.broadcast_arrays(np.asarray(lo, float), np.asarray(hi, float), np.asarray(T, float))
    C2, conc, sigdpi = 1.438786, 15.0 / math.pi ** 4, 5.67032e-8 / math.pi
    cold = T < 1e-4
    Ts = np.where(cold, 1.0, T)
    v0, v1 = C2 * lo / Ts, C2 * hi / Ts
    f = lambda v: v ** 3 / np.expm1(np.minimum(v, 700.0))  # noqa: E731
    old, done = np.zeros_like(v0), np.zeros(v0.shape, dtype=bool)
    simpson = np.zeros_like(v0)
    for n in range(1, 11):
        h = (v1 - v0) / (2.0 * n)
        val = f(v0) + f(v1)
        for k in range(1, 2 * n):
            val = val + 2.0 * (1 + k % 2) * f(v0 + k * h)
        val = val * h / 3.0
        simpson = np.where(done, simpson, val)
        with np.errstate(invalid="ignore", divide="ignore"):
            done |= np.abs((val - old) / val) <= 1e-6
        old = val
        if done.all():
            break

    def series(v):
        vs = v * v
        small = conc * vs * v * (1 / 3 + v * (-1 / 8 + v * (1 / 60 + vs * (-1 / 5040 + vs * (1 / 272160 - vs / 13305600)))))
        terms = 1 + sum((v < q).astype(int) for q in (10.25, 5.7, 3.9, 2.9, 2.3, 1.9))
        big = np.zeros_like(v)
        for m in range(1, 8):
            mv = m * v
            big += np.where(m <= terms, np.exp(-mv) * (6 + mv * (6 + mv * (3 + mv))) / m ** 4, 0.0)
        return v < 1.5, small, conc * big

    s0, p0, d0 = series(v0)
    s1, p1, d1 = series(v1)
    wide = np.where(s0 & s1, p1 - p0, np.where(s0, 1.0 - p0 - d1, d0 - d1))
    out = np.where((hi - lo) / hi < 1e-2, conc * simpson, wide) * sigdpi * Ts ** 4
    return np.where(cold, 0.0, out)


def _planck_dT(lo, hi, T):
    C2, conc, sigdpi = 1.438786, 15.0 / math.pi ** 4, 5.67032e-8 / math.pi
    v0, v1 = C2 * lo / T, C2 * hi / T
    f = lambda v: v ** 3 / np.expm1(v)  # noqa: E731
    return 4.0 * _planck(lo, hi, T) / T - sigdpi * conc * T ** 3 * (v1 * f(v1) - v0 * f(v0))


def _legendre(m, x, count):
    """Normalised P_l^m(x), l = 0..count-1: [count, len(x)]."""
    x = torch.as_tensor(x, dtype=torch.float64)
    y = torch.zeros((count,) + x.shape, dtype=torch.float64)
    pmm = torch.ones_like(x)
    for k in range(1, m + 1):
        pmm = -torch.sqrt((1.0 - 1.0 / (2.0 * k)) * (1.0 - x * x)) * pmm
    if m < count:
        y[m] = pmm
    if m + 1 < count:
        y[m + 1] = math.sqrt(2.0 * m + 1.0) * x * pmm
    for k in range(m + 2, count):
        a, b = math.sqrt((k - m) * (k + m)), math.sqrt((k - m - 1) * (k + m - 1))
        y[k] = ((2.0 * k - 1.0) * x * y[k - 1] - b * y[k - 2]) / a
    return y


def _columns(N, q, modes, R=None, radiance=None):
    """Columns of N streams, arrays q: dtau, ssa, mom [I, L, >= N + 2], alb, mu0, fbeam [I], level Planck values
    planck [I, L+1, R] and pbot [I, R] (or None), dmplus, L [I] (layer counts; layers past them are ignored),
    tau [I, T] output depths (None: the levels).  Returns {field: [I, T, R]} and, with radiance =
    (mu, phi), intensities."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda a: torch.as_tensor(a, dtype=torch.float64).to(dev)  # noqa: E731
    h = N // 2
    xg, wg = np.polynomial.legendre.leggauss(h)
    mu, w = t(0.5 * (1.0 + xg)), t(0.5 * wg)
    mus = torch.cat([mu, -mu])
    w2 = torch.cat([w, w])
    dtau, ssa, mom = t(q["dtau"]), t(q["ssa"]), t(q["mom"])
    I, L = dtau.shape
    live = torch.arange(L, device=dev)[None, :] < torch.as_tensor(q["L"], device=dev)[:, None]
    thermal = q.get("planck") is not None
    R = 1 if not thermal else q["planck"].shape[-1]
    fb, mu0, alb = t(q["fbeam"]), t(q["mu0"]), t(q["alb"])
    # delta-M / delta-M+ scaling
    pN, pN1 = mom[..., N], mom[..., N + 1] if mom.shape[-1] > N + 1 else mom[..., N]
    dm = ((pN != 0) & live).any(1)
    plus = torch.zeros_like(dm)
    if q["dmplus"]:
        plus = ~(((pN < 1e-4) | (pN1 < 0.7 * pN)) & live).any(1)
    safe = lambda v: torch.where(v > 0, v, torch.full_like(v, 0.5))  # noqa: E731
    sig = ((N + 1.0) ** 2 - N * N) / (2.0 * (torch.log(safe(pN)) - torch.log(safe(pN1))))
    use_sig = plus[:, None] & ~((mom[..., N - 1] == pN) | (pN == pN1))
    f = torch.where(use_sig, torch.exp(N * N / (2.0 * sig)) * pN, torch.where((dm | plus)[:, None], pN, torch.zeros_like(pN)))
    k = torch.arange(N, dtype=torch.float64, device=dev)
    cut = torch.where(use_sig[..., None], torch.exp(-k * k / (2.0 * sig[..., None])), torch.ones_like(k))
    ws = ssa * (1.0 - f) / (1.0 - f * ssa)
    dts = (1.0 - f * ssa) * dtau
    g = (2.0 * k + 1.0) * ws[..., None] * (mom[..., :N] - f[..., None] * cut) / (1.0 - f[..., None])
    zero = torch.zeros((I, 1), dtype=torch.float64, device=dev)
    tc = torch.cat([zero, torch.cumsum(torch.where(live, dtau, 0 * dtau), 1)], 1)
    ts = torch.cat([zero, torch.cumsum(torch.where(live, dts, 0 * dts), 1)], 1)
    absorbed = torch.cat([zero, torch.cumsum(torch.where(live, (1.0 - ssa) * dtau, 0 * dtau), 1)], 1)
    Lc = torch.as_tensor(q["L"], device=dev)
    nabs = ((absorbed[:, :-1] < 10.0) & live).sum(1)
    cutoff = (absorbed[:, -1] >= 10.0) & (Lc > 1) & (not thermal)
    ncut = torch.where(cutoff, nabs, Lc)
    T = torch.exp(-ts / mu0[:, None]) * (torch.arange(L + 1, device=dev)[None, :] <= nabs[:, None]) * (fb > 0)[:, None]
    M = len(modes)
    Y = torch.stack([_legendre(m, mus.cpu(), N) for m in modes]).to(dev)  # [M, l, N]
    Y0 = torch.stack([_legendre(m, -mu0.cpu(), N) for m in modes]).to(dev)  # [M, l, I]
    par = torch.tensor([[(l + m) % 2 for l in range(N)] for m in modes], device=dev)
    eye = torch.eye(h, dtype=torch.float64, device=dev)

    def sums(sel):  # sum over one parity of g_l P_l(mu_i) P_l(mu_j): [M, I, L, h, h]
        Yp = Y[:, :, :h] * (par == sel)[:, :, None]
        return torch.einsum("ilk,mkab->milab", g, torch.einsum("mka,mkb->mkab", Yp, Yp))

    odd, even = sums(1), sums(0)
    d = torch.sqrt(w * mu)
    A = -((odd * w - eye) / mu[:, None])  # -(alpha - beta)
    B = -((even * w - eye) / mu[:, None])
    As, Bs = d[:, None] * A / d, d[:, None] * B / d
    sym = lambda X: 0.5 * (X + X.transpose(-1, -2))  # noqa: E731
    C = torch.linalg.cholesky(sym(As))
    S = sym(C.transpose(-1, -2) @ sym(Bs) @ C).reshape(-1, h, h)
    pairs = [torch.linalg.eigh(part) for part in S.split(16384)]
    lam = torch.cat([a for a, _ in pairs]).reshape(M, I, L, h)
    V = torch.cat([b for _, b in pairs]).reshape(M, I, L, h, h)
    kk = torch.sqrt(lam)  # [M, I, L, h]
    Em = torch.linalg.solve_triangular(C.transpose(-1, -2), V, upper=True) / d[:, None]
    Ep = -(A @ Em) / kk[..., None, :]
    P, Q = 0.5 * (Ep + Em), 0.5 * (Ep - Em)
    E = torch.exp(-kk * dts[None, :, :, None])
    # particular solutions (up, down) [M, I, L, N]
    phase = 0.5 * torch.einsum("ilk,mkab->milab", g, torch.einsum("mka,mkb->mkab", Y, Y)) * w2
    fac = torch.tensor([1.0 if m == 0 else 2.0 for m in modes], dtype=torch.float64, device=dev)
    full = torch.eye(N, dtype=torch.float64, device=dev)
    zb = torch.zeros((M, I, L, N), dtype=torch.float64, device=dev)
    if bool((fb > 0).any()):
        src = torch.einsum("ilk,mka,mki->mila", g, Y, Y0) * (fac[:, None] * fb[None, :])[:, :, None, None] / (4.0 * math.pi)
        zb = torch.linalg.solve(full * (1.0 + mus[None, None, :] / mu0[:, None, None])[None, :, None] - phase, src[..., None])[..., 0]
    z0 = z1 = None
    if thermal:
        B0, B1 = t(q["planck"])[:, :-1], t(q["planck"])[:, 1:]
        xr1 = torch.where((dts > 1e-4)[..., None], (B1 - B0) / dts[..., None], 0 * B0)  # [I, L, R]
        xr0 = B0 - xr1 * ts[:, :-1, None]
        one = torch.ones((I, L, N, 1), dtype=torch.float64, device=dev) * (1.0 - ws)[..., None, None]
        u = torch.linalg.solve(full - phase[0], one)  # mode 0 comes first
        v = torch.linalg.solve(full - phase[0], mus[:, None] * u)
        z1 = u * xr1[:, :, None, :]
        z0 = u * xr0[:, :, None, :] + v * xr1[:, :, None, :]

    def particular(l, tau, trans):  # [M, I, N, R] of layer l at scaled depth tau [I], beam factor trans [I]
        z = (zb[:, :, l] * trans[None, :, None])[..., None].expand(M, I, N, R).clone()
        if thermal:
            z[0] += z0[:, l] + z1[:, l] * tau[:, None, None]
        return z

    rho = torch.zeros((M, I, h, h), dtype=torch.float64, device=dev)
    s = torch.zeros((M, I, h, R), dtype=torch.float64, device=dev)
    kept = []
    for l in range(L):
        Pl, Ql, El = P[:, :, l], Q[:, :, l], E[:, :, l]
        zt, zbm = particular(l, ts[:, l], T[:, l]), particular(l, ts[:, l + 1], T[:, l + 1])
        rhs = torch.cat([(rho @ Ql - Pl) * El[..., None, :], rho @ zt[..., :h, :] - zt[..., h:, :] + s], -1)
        sol = torch.linalg.solve(Ql - rho @ Pl, rhs)
        a1, a0 = sol[..., :h], sol[..., h:]
        PE, QE = Pl * El[..., None, :], Ql * El[..., None, :]
        U, D = PE @ a1 + Ql, QE @ a1 + Pl
        u0, d0 = PE @ a0 + zbm[..., :h, :], QE @ a0 + zbm[..., h:, :]
        new = torch.linalg.solve(U.transpose(-1, -2), D.transpose(-1, -2)).transpose(-1, -2)
        go = (l < ncut)[None, :, None, None]
        s = torch.where(go, d0 - new @ u0, s)
        rho = torch.where(go, new, rho)
        kept.append((a1, a0, U, u0))
    # surface: up = 2 alb sum w mu down + sources
    m0 = (torch.tensor(list(modes), device=dev) == 0).double()
    lit = m0[:, None] * torch.where(cutoff, 0 * alb, alb)[None, :]
    refl = 2.0 * lit[..., None, None] * (w * mu)[None, None, None, :].expand(M, I, h, h)
    ground = (lit * (mu0 * fb / math.pi * T.gather(1, Lc[:, None])[:, 0])[None])[..., None, None].expand(M, I, h, R).clone()
    if thermal:
        ground[0] += ((1.0 - alb)[:, None] * t(q["pbot"]))[:, None, :]
    up = torch.linalg.solve(torch.eye(h, dtype=torch.float64, device=dev) - refl @ rho, refl @ s + ground)
    ca = torch.zeros((M, I, L, h, R), dtype=torch.float64, device=dev)
    cb = torch.zeros_like(ca)
    bottom = up
    for l in range(L - 1, -1, -1):
        a1, a0, U, u0 = kept[l]
        up = torch.where((l == ncut - 1)[None, :, None, None], bottom, up)
        b = torch.linalg.solve(U, up - u0)
        a = a1 @ b + a0
        go = (l < ncut)[None, :, None, None]
        ca[:, :, l], cb[:, :, l] = torch.where(go, a, 0 * a), torch.where(go, b, 0 * b)
        zt = particular(l, ts[:, l], T[:, l])
        up = torch.where(go, P[:, :, l] @ a + (Q[:, :, l] * E[:, :, l, None, :]) @ b + zt[..., :h, :], up)
    # output depths, their layers
    if q.get("tau") is None:
        lay = torch.cat([torch.zeros(1, dtype=torch.long), torch.arange(L)]).to(dev)[None].expand(I, L + 1)
        ut, us = tc, ts
        beyond = torch.arange(L + 1, device=dev)[None] > ncut[:, None]
    else:
        ut = t(q["tau"])
        inside = (ut[:, :, None] >= tc[:, None, :-1]) & (ut[:, :, None] <= tc[:, None, 1:]) & live[:, None, :]
        lay = torch.where(inside.any(2), inside.double().argmax(2), (Lc - 1)[:, None])
        at = lambda a: a.gather(1, lay)  # noqa: E731
        us = at(ts) + (1.0 - at(ssa * f)) * (ut - at(tc))
        beyond = lay >= ncut[:, None]
    nT = ut.shape[1]
    at = lambda a: a.gather(1, lay)  # noqa: E731

    def pick(a):  # layer array [I, L, ...] at the output layers
        return a[torch.arange(I, device=dev)[:, None], lay]

    top, bot = at(ts[:, :-1]), at(ts[:, 1:])
    ea = torch.exp(-pick(kk[0]) * (us - top)[..., None])[..., None] * pick(ca[0])
    eb = torch.exp(-pick(kk[0]) * (bot - us)[..., None])[..., None] * pick(cb[0])
    dirf = torch.where(fb[:, None] > 0, torch.exp(-us / mu0[:, None]), 0 * us)
    z = (pick(zb[0]) * dirf[..., None])[..., None].expand(I, nT, N, R).clone()
    if thermal:
        z += pick(z0) + pick(z1) * us[..., None, None]
    Iu = pick(P[0]) @ ea + pick(Q[0]) @ eb + z[..., :h, :]
    Id = pick(Q[0]) @ ea + pick(P[0]) @ eb + z[..., h:, :]
    tot = lambda X, v: torch.einsum("itar,a->itr", X, v)  # noqa: E731
    two = 2.0 * math.pi
    direct = (fb[:, None] * dirf)[..., None].expand(I, nT, R)
    fdir = ((mu0 * fb)[:, None] * torch.where(fb[:, None] > 0, torch.exp(-ut / mu0[:, None]), 0 * ut))[..., None].expand(I, nT, R)
    md, mup = two * tot(Id, w) / (4 * math.pi), two * tot(Iu, w) / (4 * math.pi)
    mean = md + mup + direct / (4 * math.pi)
    plk = pick(xr0) + pick(xr1) * us[..., None] if thermal else 0.0
    out = dict(flux_direct_beam=fdir, flux_down=two * tot(Id, w * mu) + mu0[:, None, None] * direct - fdir,
               flux_up=two * tot(Iu, w * mu), flux_tau_divergence=(1.0 - at(ssa))[..., None] * 4 * math.pi * (mean - plk),
               mean_intensity=mean, mean_intensity_down=md, mean_intensity_up=mup,
               mean_intensity_direct_beam=direct / (4 * math.pi))
    out = {k2: torch.where(beyond[..., None], 0 * v, v) for k2, v in out.items()}
    if radiance is None:
        return out
    um, phi = t(radiance[0]), np.asarray(radiance[1])
    Yu = torch.stack([_legendre(m, um.cpu(), N) for m in modes]).to(dev)  # [M, l, nu]
    Tm = 0.5 * torch.einsum("ilk,mkub->milub", g, torch.einsum("mku,mkb->mkub", Yu, Y)) * w2
    GA = Tm @ torch.cat([P, Q], -2)  # [M, I, L, nu, h]
    GB = Tm @ torch.cat([Q, P], -2)
    zbu = (Tm @ zb[..., None])[..., 0] + torch.einsum("ilk,mku,mki->milu", g, Yu, Y0) * (fac[:, None] * fb[None] / (4 * math.pi))[:, :, None, None]
    ga, gb = GA * ca[..., 0][..., None, :], GB * cb[..., 0][..., None, :]
    res = torch.zeros((M, I, nT, len(um)), dtype=torch.float64, device=dev)
    lidx = torch.arange(L, device=dev)
    used = lidx[None] < ncut[:, None]
    for iu in range(len(um)):
        x = float(um[iu])
        for it in range(nT):
            tt, y = us[:, it:it + 1], lay[:, it:it + 1]
            if x > 0:
                on = used & (lidx[None] >= y)
                a0, a1 = torch.maximum(ts[:, :-1], tt), ts[:, 1:]
            else:
                on = used & (lidx[None] <= y)
                a0, a1 = ts[:, :-1], torch.minimum(ts[:, 1:], tt)
            on = on & (a1 >= a0)
            a0, a1 = torch.where(on, a0, 0 * a0), torch.where(on, a1, 0 * a1)
            e1, e2 = torch.exp(torch.where(on, (tt - a0) / x, 0 * a0)), torch.exp(torch.where(on, (tt - a1) / x, 0 * a0))
            D = a1 - a0
            amp_a = torch.exp(-kk * torch.where(on, a0 - ts[:, :-1], 0 * a0)[None, ..., None])
            amp_b = torch.exp(-kk * torch.where(on, ts[:, 1:] - a1, 0 * a0)[None, ..., None])
            ek = torch.exp(-kk * D[None, ..., None])
            sgn = 1.0 if x > 0 else -1.0
            E1, E2 = e1[None, ..., None], e2[None, ..., None]

            def ratio(near, far, den, lim):  # (near - far) / den, its limit where den is tiny
                ex = D[None, ..., None] * den / x
                flat = (ex.abs() < 0.3) & (den.abs() < 0.3)
                return torch.where(flat, lim * torch.special.expm1(ex) / torch.where(den == 0, torch.ones_like(den), den),
                                   (near - far) / torch.where(flat, torch.ones_like(den), den))

            if x > 0:
                fa = (E1 - E2 * ek) / (1.0 + x * kk)
                fbm = ratio(E1 * ek, E2, 1.0 - x * kk, E2)
            else:
                fa = -ratio(E1, E2 * ek, 1.0 + x * kk, E2 * ek)
                fbm = (E2 - E1 * ek) / (1.0 - x * kk)
            val = (ga[..., iu, :] * amp_a * fa + gb[..., iu, :] * amp_b * fbm).sum(-1)
            own = lidx[None] == y
            dir_t = torch.where(fb[:, None] > 0, torch.exp(-tt / mu0[:, None]), 0 * tt)
            Tl = torch.where(own, dir_t, T[:, :-1]) if x > 0 else T[:, :-1]
            Tr = T[:, 1:] if x > 0 else torch.where(own, dir_t, T[:, 1:])
            val = val + zbu[..., iu] * (sgn * (e1 * Tl - e2 * Tr) / (1.0 + x / mu0[:, None]))[None]
            if thermal:
                f0, f1 = sgn * (e1 - e2), sgn * ((a0 + x) * e1 - (a1 + x) * e2)
                zu0 = (Tm[0] @ z0)[..., iu, 0] + (1.0 - ws) * xr0[..., 0]
                zu1 = (Tm[0] @ z1)[..., iu, 0] + (1.0 - ws) * xr1[..., 0]
                val = val.clone()
                val[0] += zu0 * f0 + zu1 * f1
            total = (val * on[None]).sum(-1)
            if x > 0:
                endt = ts.gather(1, Lc[:, None])
                fall = torch.exp((tt - endt) / x)[:, 0]
                # the surface's reflected radiance is isotropic: any quadrature angle's
                lamb = (bottom[..., 0, 0] * m0[:, None]) * (~cutoff)[None]
                total = total + lamb * fall[None]
            res[:, :, it, iu] = torch.where(beyond[None, :, it], 0 * total, total)
    cosm = torch.stack([t(np.cos(m * phi * math.pi / 180.0)) for m in modes])  # [M, nphi]
    out["intensity_azimuth_avg"] = res[0]
    out["intensity"] = torch.einsum("mitu,mp->itup", res, cosm)
    return out


def _exact_flux(c, seed):
    n, L, N = c["n"], c["layers"], c["streams"]
    R = L + 2 if c["jacobian"] else 1
    if n * L * N * N * 8.0 * R > 6e9 and c["jacobian"] or n * L * float(N) ** 3 > 1.2e10:
        return None
    d = _flux_inputs(c, seed)
    pc = max(N, d["nmom"]) + 1
    back = (lambda a, ax: np.flip(a, ax)) if c["bottom_up"] else (lambda a, ax: a)
    temp = back(d["temp"], 0)
    step = max(1, int(2e8 / (L * N * N)) // R)
    parts = []
    for i0 in range(0, n, step):
        r = slice(i0, min(n, i0 + step))
        m = r.stop - i0
        lo, hi = d["lo"][r, None], d["hi"][r, None]
        q = dict(dtau=back(d["dtau"][r], 1).copy(), ssa=back(d["ssa"][r], 1).copy(),
                 mom=_moments(back(d["g"][r], 1).copy(), pc, "cpu"), alb=d["albedo"][r], mu0=d["mu0"][r],
                 fbeam=np.full(m, d["fbeam"]), dmplus=c["dmplus"], L=np.full(m, L))
        if c["thermal"]:
            q["planck"] = _planck(lo, hi, temp[None, :])[..., None]
            q["pbot"] = _planck(lo, hi, np.full((1, 1), temp[-1]))
        o = {k: v[..., 0] for k, v in _columns(N, q, (0,)).items()}
        if c["jacobian"]:
            unit = np.zeros((m, L + 1, R))
            unit[:, np.arange(L + 1), np.arange(L + 1)] = 1.0
            low = np.zeros((m, R))
            low[:, L + 1] = 1.0
            jq = dict(q, planck=unit, pbot=low, fbeam=np.zeros(m))
            j = _columns(N, jq, (0,))
            dT = torch.as_tensor(_planck_dT(lo, hi, np.concatenate([temp, temp[-1:]])[None, :])).to(j["flux_up"].device)
            for f in capi.JAC_FIELDS:
                v = j[capi.JAC_OF[f]] * dT[:, None, :]
                if c["bottom_up"]:
                    v = torch.flip(v, [1])
                    v = torch.cat([torch.flip(v[..., :-1], [2]), v[..., -1:]], 2)
                o["jac." + f] = v
        parts.append({k: (torch.flip(v, [1]) if c["bottom_up"] and not k.startswith("jac.") else v).cpu()
                      for k, v in o.items()})
    o = {k: torch.cat([p[k] for p in parts]) for k in parts[0]}
    res = {k: v for k, v in o.items() if not k.startswith("jac.")}
    res["status"] = None
    if c["jacobian"]:
        res["jacobians"] = {f: o["jac." + f] for f in capi.JAC_FIELDS}
    return res


def _exact_general(c, seed):
    d = _general_inputs(c, seed)
    n, N, L, off = c["n"], d["num_streams"], d["num_layers"], d["layer_offset"]
    modes = (lambda s: s) if c["beam"] else (lambda s: 1)
    if sum(modes(int(s)) * float(l) * int(s) ** 3 for s, l in zip(N, L)) > 1.2e10:
        return None
    mu, phi = _angles(c)
    out = {}
    for s in sorted(set(N.tolist())):
        group = np.flatnonzero(N == s)
        group = group[np.argsort(L[group], kind="stable")]
        step = max(1, int(1.5e8 / (modes(s) * int(L[group].max()) * s * s)))
        for g0 in range(0, len(group), step):
            ids = group[g0:g0 + step]
            Lm = int(L[ids].max())
            pad = lambda a, v: np.stack([np.concatenate([a[off[i]:off[i + 1]], np.full((Lm - L[i],) + a.shape[1:], v)]) for i in ids])  # noqa: E731
            q = dict(dtau=pad(d["delta_tau"], 0.1), ssa=pad(d["single_scat_albedo"], 0.5),
                     mom=pad(d["phase_function_moments"][:, :s + 2], 0.1), alb=d["surface_albedo"][ids],
                     mu0=d["direct_beam_mu"][ids], fbeam=d["direct_beam_flux"][ids], dmplus=c["dmplus"], L=L[ids],
                     tau=d["tau_user"][0][ids])
            if c["thermal"]:
                temp = np.stack([np.concatenate([d["temperature"][off[i] + i:off[i + 1] + i + 1], np.full(Lm - L[i], 250.0)]) for i in ids])
                lo, hi = d["wavenumber_low"][ids, None], d["wavenumber_high"][ids, None]
                q["planck"] = _planck(lo, hi, temp)[..., None]
                q["pbot"] = _planck(lo, hi, d["temperature_bottom"][ids, None])
            o = _columns(s, q, range(modes(s)), radiance=(mu, phi))
            for k, v in o.items():
                v = v.cpu().numpy()
                v = v[..., 0] if k in capi.FLUX_OUT_FIELDS else v
                out.setdefault(k, np.zeros((n,) + v.shape[1:]))[ids] = v
    return dict(out, status=None)


def _exact_single(c, seed):
    d = _one_column(c, seed)
    L, N = c["layers"], c["streams"]
    rad = c["kind"] == "radiance"
    lo, hi = np.array([[600.0]]), np.array([[610.0]])
    q = dict(dtau=d["dtau"][None], ssa=d["ssa"][None], mom=_moments(d["g"][None], N + (2 if rad else 1), "cpu"),
             alb=np.array([d["albedo"]]), mu0=np.array([d["mu0"]]), fbeam=np.array([1.0]), dmplus=rad,
             L=np.array([L]), planck=_planck(lo, hi, d["temp"][None])[..., None],
             pbot=_planck(lo, hi, d["temp"][None, -1:]))
    if rad:
        total = _column_total(d["dtau"])
        q["tau"] = np.array([[0.0, total / 2.0, total]])
    o = _columns(N, q, range(N) if rad else (0,), radiance=(MU5, PHI4) if rad else None)
    r = {f: o[f][0, :, 0].cpu().numpy() for f in capi.FLUX_OUT_FIELDS}
    if rad:
        for f in ("intensity", "intensity_azimuth_avg"):
            r[f] = o[f][0].reshape(-1).cpu().numpy()
    return r


def _exact_bands(c, seed):
    d = _bands_inputs(c, seed)
    n, L, N = c["n"], c["layers"], c["streams"]
    q = dict(dtau=d["dtau"], ssa=d["ssa"], mom=_moments(np.full((n, L), d["g"]), N + 1, "cpu"), alb=d["albedo"],
             mu0=np.full(n, d["mu0"]), fbeam=np.full(n, math.pi), dmplus=False, L=np.full(n, L))
    return {k: v[..., 0].cpu().numpy() for k, v in _columns(N, q, (0,)).items()}


def _exact_emulator(c, seed):
    params, x, y, hw = _emulator_inputs(c, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rnd = lambda a: torch.from_numpy(a).to(dev).to(torch.bfloat16).double()  # noqa: E731
    P = [(rnd(W).requires_grad_(c["training"]), torch.from_numpy(b).to(dev).double().requires_grad_(c["training"]))
         for W, b in params]
    H = rnd(x)
    for W, b in P[:-1]:
        H = torch.nn.functional.gelu(H @ W.T + b)
    out = H @ P[-1][0].T + P[-1][1]
    if not c["training"]:
        return out
    Y, HW = torch.from_numpy(y).to(dev).double(), torch.from_numpy(hw).to(dev).double()
    nh, no = EMU["n_heads"], EMU["n_out"]
    sq = (HW[:, :, None] * (out.reshape(-1, nh, no) - Y[:, None, :]) ** 2).sum()
    grads = torch.autograd.grad(sq / (no * c["rows"]), [v for pair in P for v in pair])
    flat = []
    for g in grads:
        shape = [_pad64(v) for v in g.shape]
        full = torch.zeros(shape, dtype=torch.float64, device=dev)
        full[tuple(slice(0, v) for v in g.shape)] = g
        flat.append(full.reshape(-1))
    return dict(gradients=torch.cat(flat), loss=sq.detach().reshape(1))


def exact(case, seed):
    return {"flux": _exact_flux, "general": _exact_general, "column": _exact_single, "radiance": _exact_single,
            "bands": _exact_bands, "emulator": _exact_emulator}[case["kind"]](case, seed)
