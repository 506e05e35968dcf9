"""The work that users of this package have it do, as cases: sizes, inputs, one pass through the public entry points,
the bytes and operations a pass cannot do without, and its results in plain 64-bit torch.

Eight kinds of call, each over its range of batch sizes:

* ``device``    a batch on device-resident weights and parameters (``batch_device``): a fitting loop or a sampler that
                draws on the GPU. One walker, an ensemble, a catalogue; with the diffuse screen alone or with birth
                clouds, an old-star screen, escaping light and a dust slope per model.
* ``sfh``       the delayed-tau batch from parameters alone (``csp_batch``; 20 filters, z = 0).
* ``grad``      forward and reverse for magnitude cotangents (``csp_batch_grad``) with weights over ages and
                metallicities: one step of a gradient-based fit.
* ``ops``       the batch with an IMF per model through the SSP operators, delayed-tau SFH.
* ``ops_grad``  its forward and reverse.
* ``emission``  the delayed-tau batch with nebular lines, dust emission and the AGN torus.
* ``emulator``  the learned emulator on device inputs.
* ``mags``      magnitudes of spectra already on the device (``spec_mags_noalloc``).

Spectra, magnitudes and gradients are computed in FP32 (split-BF16 products) behind the C API's doubles; a pass hands
them on as the FP32 tensors on the GPU that a likelihood or an optimiser takes. Mass and L_bol are FP64 sums and stay
FP64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from libopensps_gb300 import emulator, synth_dust, synth_ops, synthdata
from libopensps_gb300.capi import DEVICE_PARAMS, EMU_INPUTS, Context
from libopensps_gb300.torch_fn import GRAD_ROWS
from libopensps_gb300.workloads import DEVICE_PARAM_DEFAULTS

NS, NT, NZ = synthdata.NSPEC, synthdata.NT, synthdata.NZ
NTZ = NT * NZ


def listed() -> list:
    return [
        # one walker of a sampler that stays on the GPU: latency
        {"name": "walker_1", "kind": "device", "n": 1, "screens": "diffuse"},
        # an ensemble sampler's step
        {"name": "ensemble_1000", "kind": "device", "n": 1000, "screens": "diffuse"},
        # a survey field with birth clouds, an old-star screen, escaping light and a dust slope per galaxy
        {"name": "birth_clouds_9001", "kind": "device", "n": 9001, "screens": "birth_cloud"},
        # a catalogue or a training set (the benchmark's batch)
        {"name": "catalogue_65536", "kind": "device", "n": 65536, "screens": "diffuse"},
        # the delayed-tau configuration of the benchmark
        {"name": "delayed_tau_256", "kind": "sfh", "n": 256},
        # a gradient step of a hierarchical fit
        {"name": "gradient_2000", "kind": "grad", "n": 2000},
        # an IMF per model (the benchmark's operator batch)
        {"name": "imf_1024", "kind": "ops", "n": 1024},
        # gradients for a handful of chains with an IMF each
        {"name": "imf_gradient_100", "kind": "ops_grad", "n": 100},
        # every emission component, a photometric survey's field
        {"name": "emission_4001", "kind": "emission", "n": 4001},
        # the emulator inside a sampler
        {"name": "emulator_500", "kind": "emulator", "n": 500},
        # the emulator over a simulation's galaxies (the benchmark's batch)
        {"name": "emulator_1048576", "kind": "emulator", "n": 1048576},
        # photometry of spectra from elsewhere
        {"name": "photometry_20001", "kind": "mags", "n": 20001},
    ]


#: the range of batch sizes of each kind
SIZES = {"device": (1, 65536), "sfh": (1, 4096), "grad": (1, 4096), "ops": (1, 4096), "ops_grad": (1, 1024),
         "emission": (1, 8192), "emulator": (1, 1048576), "mags": (1, 65536)}


def draw(rng) -> dict:
    kind = rng.choice(sorted(SIZES))
    lo, hi = SIZES[kind]
    case = {"kind": kind, "n": max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5))))))}
    if kind == "device":
        case["screens"] = rng.choice(["diffuse", "birth_cloud"])
    return case


# ---------------------------------------------------------------------------------------------- the program's side
_contexts: dict = {}


def _context(kind: str) -> Context:
    """The context a program keeps for its calls of one kind (libraries, operators and weights are loaded once)."""
    group = {"grad": "device", "mags": "device", "ops_grad": "ops_grad"}.get(kind, kind)
    if group not in _contexts:
        if group == "emulator":
            c = emulator.training_context()
            c.emulator_load(emulator.WEIGHTS)
        else:
            c = Context()
        if group in ("device", "emission"):
            c.set_int("add_neb_emission", 1)
        if group in ("device", "emission", "ops", "ops_grad"):
            c.set_int("add_igm_absorption", 1)
        if group == "sfh":
            c.set_filters_library("gauss20")
        if group in ("sfh", "ops", "emission"):
            c.set_int("sfh", 4)
        if group in ("ops", "ops_grad"):
            c.build_ssp_ops()
        if group == "emission":
            c.set_int("add_dust_emission", 1)
            c.set_int("add_agn_dust", 1)
        _contexts[group] = c
    return _contexts[group]


def _uniform(gen, n, lo, hi):
    return torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _weights(gen, n):
    """Weights over ages and metallicities for one solar mass formed, (n, NZ, NT) on the GPU: a Dirichlet(1) history
    over the ages times a Gaussian in log Z."""
    sfh = -torch.log1p(-torch.rand((n, NT), generator=gen, device="cuda", dtype=torch.float64))
    sfh /= sfh.sum(1, keepdim=True)
    logz = torch.linspace(-2.0, 0.5, NZ, device="cuda", dtype=torch.float64)
    cen, sig = _uniform(gen, n, -2.0, 0.5), _uniform(gen, n, 0.1, 0.5)
    zw = torch.exp(-0.5 * ((logz[None] - cen[:, None]) / sig[:, None]) ** 2)
    zw /= zw.sum(1, keepdim=True)
    return (zw[:, :, None] * sfh[:, None, :]).contiguous()


def _inputs(case: dict, seed: int) -> dict:
    """A case's inputs (FP64 on the GPU): ``par`` by parameter name, ``wz`` weights, ``mags_bar`` cotangents, ``spec``."""
    kind, n = case["kind"], case["n"]
    gen = torch.Generator(device="cuda").manual_seed(seed * 1000003 + n)
    par, out = {}, {}

    def put(name, lo, hi):
        par[name] = _uniform(gen, n, lo, hi)

    if kind in ("sfh", "ops", "emission", "emulator"):
        par["tau"] = 10.0 ** _uniform(gen, n, -1.0, 1.0)
        put("tage", 1.0, 13.7)
        put("logzsol", -2.0, 0.5)
    put("dust2", 0.0, 2.0 if kind == "sfh" else 3.0)
    if kind != "sfh":
        put("zred", 0.0, 6.0)
        put("sigma_smooth", 50.0, 300.0)
    if kind == "emulator":
        put("dust_index", -1.0, -0.4)
    if kind in ("ops", "ops_grad", "emulator"):
        put("imf1", 0.3, 1.8)
        put("imf2", 1.3, 2.8)
        put("imf3", 1.8, 3.3)
    if case.get("screens") == "birth_cloud":
        put("dust1", 0.0, 2.0)
        put("dust3", 0.0, 0.4)
        put("dust_index", -1.0, -0.4)
        put("frac_obrun", 0.0, 0.3)
        put("frac_nodust", 0.0, 0.2)
    if kind == "emission":
        put("dust1", 0.1, 1.0)
        put("dust3", 0.0, 0.4)
        put("duste_qpah", 0.5, 4.5)
        put("duste_umin", 0.1, 25.0)
        put("duste_gamma", 0.0, 0.5)
        put("fagn", 0.0, 1.0)
        put("agn_tau", 5.0, 150.0)
    out["par"] = par
    if kind in ("device", "grad", "ops_grad"):
        out["wz"] = _weights(gen, n)
    if kind in ("grad", "ops_grad"):
        out["mags_bar"] = torch.randn((n, 40), generator=gen, device="cuda", dtype=torch.float64)
    if kind == "mags":
        # smooth L_nu spectra with lines' scatter, the magnitude of a galaxy's per solar mass
        x = torch.linspace(0.0, 1.0, NS, device="cuda")[None]
        a, b, c = (_uniform(gen, n, lo, hi).float()[:, None] for lo, hi in ((-6.0, 2.0), (0.2, 0.6), (0.2, 0.5)))
        noise = torch.randn((n, NS), generator=gen, device="cuda")
        out["spec"] = 1e-15 * torch.exp(a * (x - 0.5) - ((x - b) / c) ** 2 + 0.05 * noise)
    return out


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def prepare(case: dict, seed: int):
    kind, n = case["kind"], case["n"]
    ctx = _context(kind)
    inp = _inputs(case, seed)
    par = inp["par"]
    s = {"case": case, "ctx": ctx}
    if kind == "device":
        cols = [par.get(k, torch.full((n,), DEVICE_PARAM_DEFAULTS[k], device="cuda", dtype=torch.float64))
                for k in DEVICE_PARAMS]
        s["d_par"] = torch.stack(cols, 1).contiguous()
        s["d_wz"] = inp["wz"]
        s["d_mags"] = torch.empty((n, ctx.nbands), device="cuda", dtype=torch.float64)
        s["stream"] = torch.cuda.ExternalStream(ctx.stream())
    elif kind == "mags":
        s["d_spec"], s["d_zred"] = inp["spec"], par["zred"].contiguous()
        s["d_mags"] = torch.empty((n, ctx.nbands), device="cuda", dtype=torch.float64)
        s["stream"] = torch.cuda.ExternalStream(ctx.stream())
    elif kind == "emulator":
        s["d_x"] = torch.stack([par[k] for k in EMU_INPUTS], 1).float().contiguous()
        s["d_mags"] = torch.empty((n, ctx.nbands), device="cuda")
        s["d_pca"] = torch.empty((n, 64), device="cuda")
        s["d_spread"] = torch.empty(n, device="cuda")
        s["d_flag"] = torch.empty(n, device="cuda", dtype=torch.int32)
        s["d_flagged"] = torch.empty(n, device="cuda", dtype=torch.int32)
    else:
        s["par"] = {k: v.cpu().numpy() for k, v in par.items()}
        if kind in ("grad", "ops_grad"):
            wz, bar = _pinned((n, NZ, NT)), _pinned((n, ctx.nbands))
            wz[:], bar[:] = inp["wz"].cpu().numpy(), inp["mags_bar"].cpu().numpy()
            s["wz"], s["mags_bar"] = wz, bar
            s["out"] = {"mags": _pinned((n, ctx.nbands)), "mass": _pinned(n), "lbol": _pinned(n),
                        "params_bar": _pinned((n, 44)), "weights_z_bar": _pinned((n, NZ, NT))}
    torch.cuda.synchronize()
    return s


class _DeviceArray:
    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _spectra(ctx):
    """The last batch's spectra where they are: the context's device buffer."""
    ptr, ns, n, _ = ctx.spec_device()
    return torch.as_tensor(_DeviceArray(ptr, (n, ns), "<f4"), device="cuda")


def _f32(a):
    return torch.from_numpy(a).cuda(non_blocking=True).float()


def run(state):
    ctx, case = state["ctx"], state["case"]
    kind, n = case["kind"], case["n"]
    if kind == "device":
        ctx.batch_device(n, state["d_par"].data_ptr(), state["d_wz"].data_ptr(), state["d_mags"].data_ptr(), sync=False)
        with torch.cuda.stream(state["stream"]):
            mags = state["d_mags"].float()
        return {"mags": mags, "spec": _spectra(ctx)}
    if kind == "mags":
        ctx.spec_mags_noalloc(n, state["d_spec"].data_ptr(), state["d_zred"].data_ptr(), state["d_mags"].data_ptr(),
                              sync=False)
        with torch.cuda.stream(state["stream"]):
            return {"mags": state["d_mags"].float()}
    if kind == "emulator":
        # (the flags follow from the spread and the box; the flagged models' list is in no fixed order)
        ctx.emulator_predict_device(n, state["d_x"].data_ptr(), state["d_mags"].data_ptr(), state["d_flag"].data_ptr(),
                                    state["d_flagged"].data_ptr(), state["d_pca"].data_ptr(),
                                    state["d_spread"].data_ptr(), count=False, sync=False)
        return {"mags": state["d_mags"], "pca": state["d_pca"], "spread": state["d_spread"]}
    if kind in ("grad", "ops_grad"):
        r = ctx.csp_batch_grad(state["par"], state["wz"], mags_bar=state["mags_bar"], spec=False, out=state["out"])
        return {"mags": _f32(r["mags"]), "mass": r["mass"], "lbol": r["lbol"], "params_bar": _f32(r["params_bar"]),
                "weights_z_bar": _f32(r["weights_z_bar"])}
    r = ctx.csp_batch(state["par"], spec=False)
    return {"mags": _f32(r["mags"]), "mass": r["mass"], "lbol": r["lbol"], "spec": _spectra(ctx)}


def work(case: dict) -> dict:
    """Each input read and each output written once; the operations of the linear algebra (multiply and add), and 60
    per pixel for the screens, the IGM and the smoothing."""
    kind, n = case["kind"], case["n"]
    basis = 8.0 * NS * NTZ                                            # as split BF16 or FP32: 4 bytes; FP64 source: 8
    nb = 20 if kind == "sfh" else 40
    out = n * (8.0 * nb + 4.0 * NS)
    csp = n * (2.0 * NS * NTZ + 60.0 * NS + 2.0 * nb * NS)
    if kind == "device":
        return {"bytes": basis / 2 + n * (8.0 * NTZ + 8.0 * len(DEVICE_PARAMS)) + out, "flops": csp}
    if kind == "sfh":
        return {"bytes": basis / 2 + out, "flops": csp}
    if kind == "emission":
        return {"bytes": basis / 2 + 4.0 * NS * (7 * 44 + 9) + out, "flops": csp + n * 40.0 * NS}
    if kind == "grad":
        return {"bytes": basis / 2 + n * 2 * 8.0 * NTZ + n * 8.0 * (2 * nb + 44), "flops": 3.0 * csp}
    if kind in ("ops", "ops_grad"):
        # per model: its template weights from every isochrone point (1500 per grid point, four templates each), then
        # the library product
        pts = NTZ * synth_ops.NPT
        fold = n * (2.0 * 4 * pts + 2.0 * 2 * synth_ops.NTEMPL * NS)
        bytes_ = pts * (8.0 + 4 * 6.0 + 8.0) + 4.0 * synth_ops.NTEMPL * NS
        if kind == "ops":
            return {"bytes": bytes_ + out, "flops": fold}
        return {"bytes": bytes_ + n * 2 * 8.0 * NTZ + n * 8.0 * (2 * nb + 44), "flops": 3.0 * fold}
    if kind == "emulator":
        w = 5 * (512 * 12 + 3 * 512 * 512 + 128 * 512)
        return {"bytes": 2.0 * w + n * 4.0 * (10 + nb + 64 + 3), "flops": 2.0 * w * n}
    return {"bytes": n * (4.0 * NS + 8.0 + 8.0 * nb), "flops": n * 2.0 * nb * NS}


# ---------------------------------------------------------------------------------------------- in 64 bits
# The same quantities from the same tables in plain FP64 torch: weights (SFH by quadrature), age sums, screens, dust
# emission, IGM (Madau 1995), AGN torus, velocity smoothing, observed frame, band fluxes and AB magnitudes; gradients
# by autograd.
C_LIGHT = 2.99792458e18
LY_WAVE = (1215.67, 1025.72, 972.537, 949.743, 937.803, 930.748, 926.226, 923.150, 920.963, 919.352, 918.129, 917.181,
           916.429, 915.824, 915.329, 914.919, 914.576)
LY_COEF = (0.0036, 0.0017, 0.0011846, 0.0009410, 0.0007960, 0.0006967, 0.0006236, 0.0005665, 0.0005200, 0.0004817,
           0.0004487, 0.0004200, 0.0003947, 0.000372, 0.000352, 0.0003334, 0.00031644)
DEFAULTS = dict(DEVICE_PARAM_DEFAULTS, imf1=1.3, imf2=2.3, imf3=2.3)
_tables: dict = {}


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _grid(neb: bool, nb: int) -> dict:
    key = (neb, nb)
    if key in _tables:
        return _tables[key]
    d = synthdata.load()
    lam, ages = d["lambda"], d["log_age"]
    basis = d["ssp_spec"].reshape(NTZ, NS).copy()                     # row z NT + t
    nyoung = int(np.sum(ages <= 7.0))
    wh = int(np.sum(lam <= 912.0))
    lum = d["line_lum"]                                               # (NZ, NT, lines)
    neb_age = np.nonzero((lum != 0).any(axis=(0, 2)))[0].max() + 1
    ion = basis.reshape(NZ, NT, NS)[:, :neb_age, :wh].copy()
    if neb:
        basis.reshape(NZ, NT, NS)[:, :neb_age, :wh] = 0.0
        for i, pos in enumerate(d["line_lambda"]):
            j = min(max(int(np.sum(lam <= pos)), 1), NS - 1)
            sig = 2.0 * (lam[j] - lam[j - 1])
            prof = np.exp(-0.5 * ((lam - pos) / sig) ** 2) / (math.sqrt(2.0 * math.pi) * sig) * (pos * pos / C_LIGHT)
            prof[prof <= 1e-14 * max(prof[j - 1], prof[j])] = 0.0
            basis += lum[:, :, i].reshape(NTZ, 1) * prof
    dl = np.diff(lam)
    w = np.zeros(NS)
    w[1:] += 0.5 * dl
    w[:-1] += 0.5 * dl
    igm = np.zeros((6, NS))
    for wave, coef in zip(LY_WAVE, LY_COEF):
        igm[0] += np.where(lam < wave, coef * (lam / wave) ** 3.46, 0.0)
    igm[1] = np.where(lam < LY_WAVE[0], 0.0017 * (lam / LY_WAVE[0]) ** 1.68, 0.0)
    x, cut = lam / 911.75, lam < 911.75
    igm[2] = np.where(cut, 0.25 * x ** 3 * (1 - x ** 0.46), 0.0)
    igm[3] = np.where(cut, 9.4 * x ** 1.5 * (1 - x ** 0.18), 0.0)
    igm[4] = np.where(cut, -0.7 * x ** 3 * (x ** -1.32 - 1), 0.0)
    igm[5] = np.where(cut, -0.023 * (1 - x ** 1.68), 0.0)
    # luminosity distance at 500 scale factors [pc]
    a = np.arange(500) / 499.0 * (1.0 - 1.0 / 1001.0) + 1.0 / 1001.0
    zt = 1.0 / a - 1.0
    e = 1.0 / np.sqrt(0.27 * (1.0 + zt[:, None] * np.linspace(0.0, 1.0, 10000)[None]) ** 3 + 0.73)
    dist = (1.0 + zt) * (C_LIGHT * 1e-13 / 72.0 * 1e6) * zt / 9999.0 * (e.sum(1) - 0.5 * (e[:, 0] + e[:, -1]))
    pc = 648000.0 / math.pi * 1.495978707e13
    g = {"lam": _t(lam), "ltab": _t(np.log(lam / 5500.0)), "lage": _t(ages), "basis": _t(basis), "ion": _t(ion),
         "neb_age": int(neb_age), "wh": wh, "nyoung": nyoung, "h": math.log(lam[-1] / lam[0]) / (NS - 1),
         "mass": _t(d["ssp_mass"]), "lbol": _t(d["ssp_lbol"]), "lz": _t(np.log10(d["zlegend"] / synthdata.ZSOL)),
         "bands": _t((d[f"filters_{nb}"] * w / lam).T), "igm": _t(igm), "jtop": int(np.sum(lam < LY_WAVE[0])),
         "zt": _t(zt), "dl": _t(dist), "zp": 48.60 + 2.5 * math.log10(3.828e33 / (4.0 * math.pi * (10.0 * pc) ** 2)),
         "wnu": _t(0.5 * np.concatenate([[0.0], np.abs(np.diff(C_LIGHT / lam))]))}
    _tables[key] = g
    return g


def _delayed_tau(g, par):
    """Mass formed per age (n, NT) for SFR ~ t exp(-t / tau) since the start, linear in log age between the grid's
    ages, normalised; 32-point Gauss-Legendre in each log-age interval."""
    x, gw = np.polynomial.legendre.leggauss(32)
    x, gw = _t(x), _t(gw)
    tage, tau = par["tage"][:, None, None] * 1e9, par["tau"][:, None, None] * 1e9
    lt = torch.log10(par["tage"] * 1e9)[:, None]
    edge = torch.cat([torch.zeros(1, device="cuda", dtype=torch.float64), g["lage"]])
    lo, hi = torch.minimum(edge[:-1][None], lt), torch.minimum(edge[1:][None], lt)
    # (the first interval, from one year: split for the rule's sake at the decades)
    w = torch.zeros((lt.shape[0], NT), device="cuda", dtype=torch.float64)

    def mass(a, b):
        u = 0.5 * (a + b)[:, :, None] + 0.5 * (b - a)[:, :, None] * x
        t = 10.0 ** u
        f = (tage - t) * torch.exp((t - tage) / tau) * t * gw * (0.5 * math.log(10.0)) * (b - a)[:, :, None]
        return u, f

    dec = torch.linspace(0.0, float(g["lage"][0]), 12, device="cuda", dtype=torch.float64)
    _, f = mass(torch.minimum(dec[:-1][None], lt), torch.minimum(dec[1:][None], lt))
    w[:, 0] += f.sum((1, 2))
    u, f = mass(lo[:, 1:], hi[:, 1:])
    up = (u - g["lage"][:-1][None, :, None]) / (g["lage"][1:] - g["lage"][:-1])[None, :, None]
    w[:, :-1] += ((1.0 - up) * f).sum(2)
    w[:, 1:] += (up * f).sum(2)
    return w / w.sum(1, keepdim=True)


def _blend(g, par, w):
    """Weights over metallicities and ages at logzsol, and the linear L_bol blended in log."""
    z = par["logzsol"]
    k = (torch.searchsorted(g["lz"], z, right=True) - 1).clamp(0, NZ - 2)
    f = ((z - g["lz"][k]) / (g["lz"][k + 1] - g["lz"][k]))[:, None]
    wz = torch.zeros((z.numel(), NZ, NT), device="cuda", dtype=torch.float64)
    m = torch.arange(z.numel(), device="cuda")
    wz[m, k] = (1.0 - f) * w
    wz[m, k + 1] = f * w
    return wz, (w * 10.0 ** ((1.0 - f) * g["lbol"][k] + f * g["lbol"][k + 1])).sum(1)


def _age_sums(g, wz, fesc=None):
    n, ny = wz.shape[0], g["nyoung"]
    b = g["basis"].view(NZ, NT, NS)
    y = wz[:, :, :ny].reshape(n, -1) @ b[:, :ny].reshape(-1, NS)
    o = wz[:, :, ny:].reshape(n, -1) @ b[:, ny:].reshape(-1, NS)
    if fesc is not None:
        na, wh = g["neb_age"], g["wh"]
        for k0, k1, col in ((0, min(na, ny), y), (ny, na, o)):
            if k1 > k0:
                add = (wz[:, :, k0:k1].reshape(n, -1) @ g["ion"][:, k0:k1].reshape(-1, wh)) * fesc[:, None]
                pad = torch.nn.functional.pad(add, (0, NS - wh))
                if col is y:
                    y = y + pad
                else:
                    o = o + pad
    return y, o


def _spectrum(g, y, o, p, igm=True, emission=None, lsum=None):
    """The rest-frame spectrum: screens, dust emission, IGM, AGN torus, velocity smoothing."""
    col = lambda k: p[k][:, None]  # noqa: E731
    lam, ltab = g["lam"], g["ltab"]
    curve = torch.exp(col("dust_index") * ltab)
    tau_b, tau_o, tau_d = col("dust1") * torch.exp(col("dust1_index") * ltab), col("dust3") * curve, col("dust2") * curve
    tb, to, td = torch.exp(-tau_b), torch.exp(-tau_o), torch.exp(-tau_d)
    fo, fnd = col("frac_obrun"), col("frac_nodust")
    tot = (y * (tb * (1 - fo) + fo) + o * to) * (td * (1 - fnd) + fnd)
    if emission is not None:
        ab = y * ((1 - fo) * -torch.expm1(-tau_b) + (tb * (1 - fo) + fo) * (1 - fnd) * -torch.expm1(-tau_d)) + \
            o * (-torch.expm1(-tau_o) + to * (1 - fnd) * -torch.expm1(-tau_d))
        iq, wq = _cell(emission["qpah"], p["duste_qpah"])
        iu, wu = _cell(emission["umin"], p["duste_umin"])
        t, gam = emission["dustem"], col("duste_gamma")
        mix = lambda c: ((1 - wq) * (1 - wu) * t[2 * iu + c, iq] + wq * (1 - wu) * t[2 * iu + c, iq + 1] +  # noqa: E731
                         wq * wu * t[2 * iu + 2 + c, iq + 1] + (1 - wq) * wu * t[2 * iu + 2 + c, iq])
        esc = ((1 - gam) * mix(0) + gam * mix(1)).clamp_min(np.finfo(np.float64).tiny) * td
        wnu = g["wnu"][1:]
        tot = tot + esc * (((ab[:, 1:] + ab[:, :-1]) @ wnu) / ((esc[:, 1:] + esc[:, :-1]) @ wnu))[:, None]
    if igm:
        opz = 1.0 + p["zred"]
        b = torch.stack([opz ** q for q in (3.46, 1.68, 3.46, 1.68, 1.68, 1.68)], 1)
        tau = b @ g["igm"]
        top = tau[:, :g["jtop"]]
        jmax = top.argmax(1, keepdim=True)
        pix = torch.arange(NS, device="cuda")[None]
        tau = torch.where(pix < jmax, top.gather(1, jmax), tau)
        tot = tot * torch.where((pix < g["jtop"]) & (col("zred") > 0), torch.exp(-tau * col("igm_factor")), torch.ones_like(tau))
    if emission is not None:
        it, wt = _cell(emission["tau"], p["agn_tau"])
        s = emission["agnspec"]
        tot = tot + (p["fagn"] * lsum)[:, None] * ((1 - wt) * s[it] + wt * s[it + 1]) * td
    # velocity smoothing over +-4 sigma windows of the log-uniform grid, 1000 - 10000 A
    h, sb = g["h"], p["sigma_smooth"] / (C_LIGHT * 1e-13)
    r = torch.ceil(4.0 * sb / h).detach()
    d = torch.arange(-4, 5, device="cuda", dtype=torch.float64)[None]
    inside = d.abs() <= r[:, None]
    left = torch.where((d > -r[:, None]) & inside, torch.exp(d * h) - torch.exp((d - 1) * h), torch.zeros_like(d))
    right = torch.where((d < r[:, None]) & inside, torch.exp((d + 1) * h) - torch.exp(d * h), torch.zeros_like(d))
    sbs = torch.where(sb > 0, sb, torch.ones_like(sb))[:, None]
    w = torch.exp(-0.5 * (d * h / sbs) ** 2) * torch.exp(-d * h) * 0.5 * (left + right)
    w = w / w.sum(1, keepdim=True).clamp_min(1e-300)
    pad = torch.nn.functional.pad(tot, (4, 4))
    sm = sum(w[:, k:k + 1] * pad[:, k:k + NS] for k in range(9))
    use = ((lam >= 1e3) & (lam <= 1e4))[None] & (sb > 0)[:, None]
    return torch.where(use, sm, tot)


def _cell(grid, x):
    i = torch.searchsorted(grid, x.contiguous(), right=True).clamp(1, grid.numel() - 1) - 1
    return i, ((x - grid[i]) / (grid[i + 1] - grid[i])).clamp(0.0, 1.0)[:, None]


def _magnitudes(g, spec, z):
    lam = g["lam"]
    target = lam[None] / (1.0 + z)[:, None]
    il = (torch.searchsorted(lam, target.detach().contiguous(), right=True) - 1).clamp(0, NS - 2)
    t = (target - lam[il]) / (lam[il + 1] - lam[il])
    s0, s1 = spec.gather(1, il), spec.gather(1, il + 1)
    obs = torch.where((z > 0)[:, None], s0 + t * (s1 - s0), spec).clamp_min(0.0)
    k = (torch.searchsorted(-g["zt"], -z.detach(), right=False) - 1).clamp(0, 498)
    dm = g["dl"][k] + (g["dl"][k + 1] - g["dl"][k]) / (g["zt"][k + 1] - g["zt"][k]) * (z - g["zt"][k])
    dd = torch.where(z > 0, 5.0 * torch.log10(dm.clamp_min(1e-300) / 10.0) - 2.5 * torch.log10(1.0 + z), torch.zeros_like(z))
    return -2.5 * torch.log10(obs @ g["bands"]) - g["zp"] + dd[:, None]


class _Fold(torch.autograd.Function):
    """Template weights V (2 x templates, n) = S X for the sparse operator S and X (points, n)."""
    @staticmethod
    def forward(ctx, x, s, st):
        ctx.st = st
        return s @ x

    @staticmethod
    def backward(ctx, g):
        return ctx.st @ g, None, None


def _operator() -> dict:
    if "ops" not in _tables:
        d = synth_ops.load()
        ny = int(np.sum(synthdata.load()["log_age"] <= 7.0))
        npt = d["mini"].shape[-1]
        q = torch.arange(NTZ * npt, device="cuda").repeat_interleave(4)
        old = (torch.arange(NTZ, device="cuda") % NT >= ny).long().repeat_interleave(4 * npt)
        e = torch.as_tensor(d["idx"].reshape(-1), device="cuda").long() + synth_ops.NTEMPL * old
        c = _t(d["coef"].reshape(-1))
        size = (2 * synth_ops.NTEMPL, NTZ * npt)
        _tables["ops"] = {"s": torch.sparse_coo_tensor(torch.stack([e, q]), c, size).to_sparse_csr(),
                          "st": torch.sparse_coo_tensor(torch.stack([q, e]), c, size[::-1]).to_sparse_csr(),
                          "lib": _t(d["lib"]), "mini": _t(d["mini"].reshape(NTZ, npt)[0]),
                          "mcur": _t(d["mcur"].reshape(NTZ, npt)), "lum": _t(d["lum"].reshape(NTZ, npt))}
        assert bool((d["mini"] == d["mini"][0, 0]).all())             # (one set of stars for every grid point)
    return _tables["ops"]


def _kroupa(p, mini):
    """Stars per isochrone point and unit mass formed, (n, points): the bins halfway between the points."""
    a = [p[k][:, None] for k in ("imf1", "imf2", "imf3")]
    c2 = 0.5 ** (a[1] - a[0])
    mid = 0.5 * (mini[1:] + mini[:-1])
    lo, hi = torch.cat([mini.new_tensor([0.08]), mid])[None], torch.cat([mid, mini[-1:]])[None]

    def integral(lo, hi, weight):
        v = 0.0
        for (s0, s1), al, c in zip(((0.08, 0.5), (0.5, 1.0), (1.0, 1e9)), a, (torch.ones_like(c2), c2, c2)):
            x0, x1 = lo.clamp(s0, s1), hi.clamp(s0, s1)
            e = 1.0 - al + weight
            v = v + torch.where(x1 > x0, c * x0 ** e * torch.expm1(e * torch.log(x1 / x0)) / e, torch.zeros_like(e))
        return v

    return integral(lo, hi, 0.0) / integral(mini.new_tensor([[0.08]]), mini.new_tensor([[120.0]]), 1.0)


def _operator_sums(p, wz):
    """Young and old age sums, mass and linear L_bol through the operator."""
    op = _operator()
    n, npt = wz.shape[0], op["mini"].numel()
    stars = _kroupa(p, op["mini"])
    w = wz.reshape(n, NTZ)
    x = (w.t()[:, None, :] * stars.t()[None]).reshape(NTZ * npt, n)
    v = _Fold.apply(x, op["s"], op["st"])
    y, o = v[:synth_ops.NTEMPL].t() @ op["lib"], v[synth_ops.NTEMPL:].t() @ op["lib"]
    return y, o, ((w @ op["mcur"]) * stars).sum(1), ((w @ op["lum"]) * stars).sum(1)


def _emulate(case, seed):
    x = torch.stack([_inputs(case, seed)["par"][k] for k in EMU_INPUTS], 1).float().double()
    raw = emulator.WEIGHTS.read_bytes()
    at = 8
    def take(count, dtype):  # noqa: E306
        nonlocal at
        v = np.frombuffer(raw, dtype=dtype, count=count, offset=at)
        at += v.nbytes
        return v
    nb = int(take(9, "<i4")[6])
    take(20, "<f8")
    par = _t(take(284, "<f4"))
    faint = float(take(2, "<f4")[1])
    bias = _t(take(5 * 2176, "<f4").reshape(5, 2176))
    w0 = _t(take(5 * 512 * 64, "<f2").reshape(5, 512, 64)[:, :, :12])
    wh, w4 = _t(take(15 * 512 * 512, "<f2").reshape(3, 5, 512, 512)), _t(take(5 * 128 * 512, "<f2").reshape(5, 128, 512))
    inc, ins, omu, osig, clk = par[:12], par[12:24], par[24:152], par[152:280], par[280:284]
    g = _grid(False, nb)
    out = {"mags": [], "pca": [], "spread": []}
    for c in x.split(65536):
        feat = [torch.log10(c[:, 0]), torch.log10(c[:, 1]), c[:, 2], c[:, 3], c[:, 4], torch.log10(1.0 + c[:, 5])]
        feat += [c[:, i] for i in range(6, 10)]
        age = torch.maximum(c[:, 1] - 2.0 * c[:, 0], 0.5 * c[:, 1])
        feat.append(torch.sin(math.pi * (9.0 + torch.log10(age) - clk[0]) / clk[1]).abs())
        feat.append(torch.sin(math.pi * (c[:, 2] - clk[2]) / clk[3]).abs())
        f = (torch.stack(feat, 1) - inc) * ins
        outs = []
        for m in range(5):
            a = torch.nn.functional.silu(f @ w0[m].t() + bias[m, :512])
            for k in range(3):
                a = torch.nn.functional.silu(a @ wh[k, m].t() + bias[m, 512 * (k + 1):512 * (k + 2)])
            outs.append(a @ w4[m].t() + bias[m, 2048:])
        o = torch.stack(outs)
        mean = omu + osig * o.mean(0)
        z = c[:, 5]
        k = (torch.searchsorted(-g["zt"], -z, right=False) - 1).clamp(0, 498)
        dm = g["dl"][k] + (g["dl"][k + 1] - g["dl"][k]) / (g["zt"][k + 1] - g["zt"][k]) * (z - g["zt"][k])
        dd = torch.where(z > 0, 5.0 * torch.log10(dm.clamp_min(1e-300) / 10.0) - 2.5 * torch.log10(1.0 + z), torch.zeros_like(z))
        mags = mean[:, 64:64 + nb] + dd[:, None]
        sd = (osig * o.std(0, unbiased=False))[:, 64:64 + nb]
        counts = mags < mags.min(1, keepdim=True).values + faint
        out["mags"].append(mags)
        out["pca"].append(mean[:, :64])
        out["spread"].append(torch.where(counts, sd, torch.zeros_like(sd)).amax(1))
    return {k: torch.cat(v) for k, v in out.items()}


def exact(case: dict, seed: int):
    kind, n = case["kind"], case["n"]
    if kind == "emulator":
        return _emulate(case, seed)
    inp = _inputs(case, seed)
    neb = kind in ("device", "grad", "mags", "emission")
    g = _grid(neb, 20 if kind == "sfh" else 40)
    if kind == "mags":
        z = inp["par"]["zred"]
        return {"mags": torch.cat([_magnitudes(g, s.double(), zz)
                                   for s, zz in zip(inp["spec"].split(2048), z.split(2048))])}
    emission = None
    if kind == "emission":
        dust, agn = synth_dust.load(), synth_dust.load_agn()
        emission = {k: _t(dust[k]) for k in ("qpah", "umin", "dustem")} | {"tau": _t(agn["tau"]), "agnspec": _t(agn["agnspec"])}
    par = {k: inp["par"].get(k, torch.full((n,), v, device="cuda", dtype=torch.float64)) for k, v in DEFAULTS.items()}
    par.update({k: v for k, v in inp["par"].items() if k not in par})
    reverse = kind in ("grad", "ops_grad")
    out = {}
    step = {"ops": 64, "ops_grad": 32, "grad": 500}.get(kind, 2048)
    for m0 in range(0, n, step):
        m = slice(m0, min(n, m0 + step))
        p = {k: v[m].clone().requires_grad_(reverse) for k, v in par.items()}
        if "wz" in inp:
            wz = inp["wz"][m].clone().requires_grad_(reverse)
            lsum = (wz * 10.0 ** g["lbol"]).sum((1, 2))
        else:
            wz, lsum = _blend(g, p, _delayed_tau(g, p))
        with torch.set_grad_enabled(reverse):
            if kind in ("ops", "ops_grad"):
                y, o, mass, lsum = _operator_sums(p, wz)
            else:
                y, o = _age_sums(g, wz, p["frac_obrun"] if neb else None)
                mass = (wz * g["mass"]).sum((1, 2))
            spec = _spectrum(g, y, o, p, igm=kind != "sfh", emission=emission, lsum=lsum)
            mags = _magnitudes(g, spec, p["zred"])
            r = {"mags": mags.detach()}
            if reverse:
                (mags * inp["mags_bar"][m]).sum().backward()
                rows = torch.zeros((wz.shape[0], 44), device="cuda", dtype=torch.float64)
                for k, row in dict(GRAD_ROWS, imf1=26, imf2=27, imf3=28).items():
                    if p[k].grad is not None:
                        rows[:, row] = p[k].grad
                r.update(params_bar=rows, weights_z_bar=wz.grad.reshape(-1, NZ, NT))
            else:
                r["spec"] = spec
            if kind != "device":
                r.update(mass=mass.detach().cpu().numpy(), lbol=torch.log10(lsum).detach().cpu().numpy())
        for k, v in r.items():
            out.setdefault(k, []).append(v)
    return {k: np.concatenate(v) if isinstance(v[0], np.ndarray) else torch.cat(v) for k, v in out.items()}
