"""The workloads this package's speed is measured on.

`listed()` names them; each stands for something a user of the operator runs, and says what. `draw(rng)` gives
further cases of the same ranges. `prepare` builds what such a program holds before the call (survey files, model,
observed data, an FwiContext or a network), `run` makes one call through the public entry points, `work` counts what
the call cannot do without, and `exact` computes the same results in 64 bits with plain torch.

The operator computes in FP32 and widens its misfit and gradients to double at the boundary; `run` hands them on in
FP32, the precision they have. Observed data are seeded records with a direct arrival and reflections of the
amplitudes the operator records, not modelled ones, so that both the package and `exact` see the same input.
"""
from __future__ import annotations

import math
import os
import shutil
import tempfile

import numpy as np
import torch

import __graft_entry__ as entry

# ---------------------------------------------------------------------------------------------------------------
# The cases. nz, nx: interior cells; pml, pad: absorbing and padding cells (pad < 0: the package's default, which
# makes the padded height a multiple of 32); nt: time steps; dx [m] sets the time step (dx / 10000 s).
# "call":
#   gradient   FwiContext.misfit_grad with the observed data in memory, all five results
#   misfit     compute_misfit of the FWI class with its gradients, observed data in the workspace's files
#   inversion  VpProblem.misfit_grad, one iteration's evaluation with model and data staged on the device
#   modelling  FwiContext.obs, the gathers of every shot
#   train, precondition   the learned preconditioner


def _fwi(name, call, nz, nx, nt, shots, *, pml=32, pad=-1, dx=10.0, aperture=0, windows=False, band=False,
         update=False, illum=False):
    return {"name": name, "call": call, "nz": nz, "nx": nx, "nt": nt, "shots": shots, "pml": pml, "pad": pad, "dx": dx,
            "aperture": aperture, "windows": windows, "band": band, "update": update, "illum": illum}


def listed():
    return [
        # A unit-test-sized gradient, the default of synthetic.tiny: nothing but launch latency.
        _fwi("tiny gradient", "gradient", 40, 60, 300, 2, pml=12, dx=20.0),
        # The reference's tutorial scale (test/TestFWI.jl's survey on a 100 x 200 model), through its FWI class.
        _fwi("layered misfit", "misfit", 100, 200, 1000, 2, dx=20.0),
        # A field-like survey of odd sizes: padded height no multiple of 32, trace windows and weights, deep
        # receivers, the 20-cell absorbing layer of small models.
        _fwi("odd windowed inversion", "inversion", 141, 317, 777, 5, pml=20, pad=7, windows=True),
        # One iteration of the learned-preconditioner family: 256 x 768 models, 16 shots, illumination on.
        _fwi("survey inversion", "inversion", 256, 768, 600, 16, illum=True),
        # Forward modelling of that survey (making observed data).
        _fwi("survey modelling", "modelling", 256, 768, 600, 16),
        # The adjoint-gradient-check model: one shot, 608 x 1600 cells.
        _fwi("single shot inversion", "inversion", 512, 1536, 2000, 1),
        # Aperture windows and uneven record lengths in one call, the benchmark's family with shorter records.
        _fwi("batched uneven inversion", "inversion", 512, 1536, 800, 24, aperture=400),
        # The full-scale model's grid, 1120 x 3152 cells.
        _fwi("large inversion", "inversion", 1024, 3072, 200, 4, pml=40, dx=5.0),
        # The band-pass option of the data path.
        _fwi("band-passed inversion", "inversion", 256, 768, 1500, 2, band=True),
        # The source-wavelet update of the data path.
        _fwi("wavelet update inversion", "inversion", 128, 384, 1000, 2, update=True),
        # One optimiser step of the preconditioner network on the 256 x 768 family (352 x 832 pixels).
        {"name": "train step", "call": "train", "nz": 352, "nx": 832},
        # Applying the network to a gradient of the 512 x 1536 model (608 x 1600 pixels).
        {"name": "precondition", "call": "precondition", "nz": 608, "nx": 1600},
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if rng.random() < 0.2:
        return {"call": rng.choice(["train", "precondition"]), "nz": 32 * spread(2, 20), "nx": spread(50, 1600)}
    call = rng.choice(["gradient", "misfit", "inversion", "inversion", "inversion", "modelling"])
    while True:
        pml = rng.choice([12, 16, 20, 32, 32, 40])
        nz, nx, nt, shots = spread(24, 1024), spread(40, 3072), spread(120, 2000), spread(1, 24)
        if call in ("gradient", "misfit"):  # through host arrays or files: the smaller models
            nz, nx, shots = min(nz, 220), min(nx, 400), min(shots, 6)
            nt = min(nt, 500) if call == "gradient" else nt
        pad = rng.choice([-1, -1, rng.randrange(0, 32)]) if call != "misfit" else -1
        cells = (nz + 2 * pml + 16) * (nx + 2 * pml)
        if 2e6 <= cells * nt * shots <= 2.5e9:
            break
    option = rng.choice(["", "", "windows", "band", "update", "illum", "aperture"]) if call == "inversion" else ""
    c = _fwi("", call, nz, nx, nt, shots, pml=pml, pad=pad, dx=rng.choice([5.0, 10.0, 20.0]),
             aperture=max(16, nx // 4) if option == "aperture" else 0, windows=option == "windows",
             band=option == "band", update=option == "update", illum=option == "illum")
    if c["band"] or c["update"]:  # these options are quadratic in the record length
        c["nt"] = min(c["nt"], 1200)
    del c["name"]
    return c


# ---------------------------------------------------------------------------------------------------------------
# Inputs.


def _random_field(shape, corr, rng):
    kz, kx = np.fft.fftfreq(shape[0])[:, None], np.fft.rfftfreq(shape[1])[None, :]
    spectrum = np.fft.rfft2(rng.standard_normal(shape)) * np.exp(-(np.pi * corr) ** 2 * (kz ** 2 + kx ** 2))
    f = np.fft.irfft2(spectrum, shape)
    f -= f.mean()
    return f / f.std()


def _wavelet(f, nt, dt):
    e, t = (np.pi * f) ** 2, dt * np.arange(nt) - 1.2 / f
    return np.cumsum((1.0 - 2.0 * e * t ** 2) * np.exp(-e * t ** 2)) * dt


def _padding(case):
    rows = case["nz"] + 2 * case["pml"]
    return 32 - rows % 32 if case["pad"] < 0 else case["pad"]


def _f0(case):
    return 100.0 / case["dx"]


def _world(case, seed):
    """Model, survey, wavelets and observed data of an FWI case."""
    rng = np.random.default_rng([int(seed), 77])
    nz, nx, pml, pad, nt, dx = (case[k] for k in ("nz", "nx", "pml", "pad", "nt", "dx"))
    pad, dt = _padding(case), dx * 1e-4
    zz, xx = np.arange(nz)[:, None], np.arange(nx)[None, :]
    dip = np.tan(np.deg2rad(rng.uniform(-5.0, 5.0)))
    cuts = np.sort(rng.uniform(0.08, 0.95, 7)) * nz
    layer = np.searchsorted(cuts, (zz - dip * (xx - nx / 2)).ravel()).reshape(nz, nx)
    vp = (1500.0 + 3000.0 * layer / 7) * (1.0 + 0.03 * np.clip(_random_field((nz, nx), 14.0, rng), -3.5, 3.5))
    vp = np.pad(vp, ((pml, pml + pad), (pml, pml)), mode="symmetric")
    shots, stf, obs = [], [], []
    for k in range(case["shots"]):
        w = nx if not case["aperture"] else int(rng.integers(min(case["aperture"], nx), nx + 1))
        xs = int(rng.integers(4, nx - 4))
        w0 = int(np.clip(xs - w // 2, 0, nx - w))
        n = nt if not case["aperture"] else int(rng.integers(3 * nt // 8, nt + 1))
        cols = np.arange(w0, w0 + w)
        rows = np.full(w, 2)
        if case["windows"]:
            rows[::7] = rng.integers(2, nz - 2, len(rows[::7]))
        s = {"z_src": 2, "x_src": xs, "z_rec": rows.tolist(), "x_rec": cols.tolist()}
        if case["aperture"]:
            s.update(nSteps=n, win_x0=w0, win_x1=w0 + w - 1)
        if case["windows"]:
            s.update(win_start=(rng.uniform(0.0, 0.2, w) * n * dt).tolist(),
                     win_end=(rng.uniform(0.6, 1.1, w) * n * dt).tolist(), weights=rng.uniform(0.5, 1.5, w).tolist())
        f = _f0(case) * (rng.uniform(0.8, 1.2) if case["aperture"] else 1.0)
        stf.append(_wavelet(f, nt, dt))
        off = np.abs(cols - xs)
        t = np.arange(n, dtype=np.float32) * np.float32(dt)
        o = np.zeros((w, n), dtype=np.float32)
        for amp, t0, v in [(1500.0, 0.0, 1550.0)] + [(rng.uniform(-120.0, 120.0), rng.uniform(0.1, 0.8) * n * dt,
                                                      rng.uniform(1800.0, 3500.0)) for _ in range(3)]:
            at = np.sqrt(t0 ** 2 + (off * dx / v) ** 2) + 1.2 / f
            tau = (t[None, :] - at[:, None].astype(np.float32)) * np.float32(np.pi * f)
            tau *= tau
            o += (amp / np.sqrt(1.0 + 0.3 * off)).astype(np.float32)[:, None] * (1.0 - 2.0 * tau) * np.exp(-tau)
        o += rng.standard_normal((w, 1), dtype=np.float32)
        obs.append(o)
        shots.append(s)
    vs, rho = vp / math.sqrt(3.0), 310.0 * vp ** 0.25
    return {"vp": vp, "vs": vs, "rho": rho, "lam": (vp * vp - 2.0 * vs * vs) * rho / 1e6, "mu": vs * vs * rho / 1e6,
            "shots": shots, "stf": np.stack(stf), "obs": obs, "pad": pad, "dt": dt}


def _mask(case, pad):
    """The inversion mask: the interior without its top 10 rows."""
    pml, nz, nx = case["pml"], case["nz"], case["nx"]
    m = np.zeros((nz + 2 * pml + pad, nx + 2 * pml))
    m[pml + 10:pml + nz, pml:pml + nx] = 1.0
    return m


def _corners(case):
    f = _f0(case)
    return [0.2 * f, 0.4 * f, 1.5 * f, 2.2 * f]


def _start_vp(case, vp):
    """What the masked-out cells hold: the evaluated model smoothed down the columns, in velocity."""
    return 0.5 * (vp + np.roll(vp, 3, axis=0))


def _net_inputs(case, seed):
    rng = np.random.default_rng([int(seed), 78])
    shape = (case["nz"], case["nx"])
    illum = np.exp(-np.arange(shape[0]) / (0.15 * shape[0]))[:, None] * np.exp(0.5 * _random_field(shape, 8.0, rng))
    grads = [s * _random_field(shape, 5.0, rng) * np.sqrt(illum) for s in (3e-2, 2e-2, 5e-1)]
    mask = np.zeros(shape)
    edge = min(32, shape[0] // 4, shape[1] // 4)
    mask[edge + 10:shape[0] - edge, edge:shape[1] - edge] = 1.0
    weights = {}
    for k, (ci, co, cip, cop) in enumerate(_LAYERS):
        w = np.zeros((9, cip, cop), dtype=np.float32)
        w[:, :ci, :co] = rng.normal(0.0, math.sqrt(2.0 / (9 * ci)) * (0.1 if k == 5 else 1.0), (9, ci, co))
        b = np.zeros(cop, dtype=np.float32)
        b[:co] = rng.normal(0.0, 0.05, co)
        weights[f"W{k}"], weights[f"b{k}"] = w, b
    return grads, illum, mask, weights


# (inputs, outputs, padded inputs, padded outputs) of the network's layers
_LAYERS = [(5, 32, 16, 32)] + [(32, 32, 32, 32)] * 4 + [(32, 3, 32, 16)]


def _features(grads, illum, mask):
    m = mask > 0
    e = np.clip(illum / illum[m].max(), 0.0, 1.0)
    scaled = [g / np.sqrt(np.mean(np.square(g[m]))) for g in grads]
    return np.stack(scaled + [e, (np.log10(np.maximum(e, 1e-6)) + 6.0) / 6.0]), e


# ---------------------------------------------------------------------------------------------------------------
# The calls.


class _Workspace:
    """A directory that lives as long as the state that holds it."""

    def __init__(self):
        self.path = tempfile.mkdtemp(prefix="fwi_case_")

    def __del__(self):
        shutil.rmtree(self.path, ignore_errors=True)


def prepare(case, seed):
    fw = entry.load_package()
    from fwiflow_gb300 import inversion, precond, utils

    call = case["call"]
    if call in ("train", "precondition"):
        grads, illum, mask, weights = _net_inputs(case, seed)
        net = precond.CnnPreconditioner(case["nz"], case["nx"], seed=0)
        net.load_state(weights)
        if call == "precondition":
            return {"call": call, "net": net, "args": (*grads, illum, mask)}
        feats, e = _features(grads, illum, mask)
        gain = np.log(1e-3 / (e + 1e-3)) * mask
        return {"call": call, "net": net, "samples": [(feats, np.stack([gain] * 3), mask)]}
    w = _world(case, seed)
    nt, dt, dx, pml, pad = case["nt"], w["dt"], case["dx"], case["pml"], w["pad"]
    work = _Workspace()
    ids = list(range(case["shots"]))
    state = {"call": call, "work": work, "stf": w["stf"], "ids": ids, "obs": w["obs"]}
    if call == "misfit":
        s = w["shots"]
        state["fwi"] = fw.FWI(case["nz"], case["nx"], dx, dx, nt, dt, f0=_f0(case), nPml=pml,
                              ind_src_z=[v["z_src"] for v in s], ind_src_x=[v["x_src"] for v in s],
                              ind_rec_z=s[0]["z_rec"], ind_rec_x=s[0]["x_rec"], workspace=work.path)
        for k, o in zip(ids, w["obs"]):
            o.tofile(os.path.join(state["fwi"].data_dir, f"Shot{k}.bin"))
        state["model"] = (w["vp"], w["vs"], w["rho"])
        vp0 = _start_vp(case, w["vp"])
        state["reference"] = (vp0, vp0 / math.sqrt(3.0), 310.0 * vp0 ** 0.25)
        return state
    para, survey = os.path.join(work.path, "para.json"), os.path.join(work.path, "survey.json")
    nz_pad, nx_pad = w["vp"].shape
    utils.paraGen(nz_pad, nx_pad, dx, dx, nt, dt, _f0(case), pml, pad, para, survey, os.path.join(work.path, "Data"),
                  if_win=case["windows"], filter_para=_corners(case) if case["band"] else None,
                  if_src_update=case["update"])
    utils.surveyGen_shots(w["shots"], survey)
    ctx = state["ctx"] = fw.FwiContext(para, 0)
    if call == "inversion":
        state["problem"] = inversion.VpProblem(ctx, w["stf"], ids, w["obs"], _start_vp(case, w["vp"]), w["vp"],
                                               _mask(case, pad))
        state["vp"], state["illum"] = w["vp"], case["illum"]
    else:
        state["model"] = (w["lam"], w["mu"], w["rho"])
    return state


def _single(v):
    return np.asarray(v, dtype=np.float32)


def run(state):
    call = state["call"]
    if call == "gradient":
        J, *grads = state["ctx"].misfit_grad(*state["model"], state["stf"], state["ids"], obs=state["obs"])
        return {"misfit": _single(J), **{k: _single(g) for k, g in zip(("lam", "mu", "den", "stf"), grads)}}
    if call == "misfit":
        fw = entry.load_package()
        cp0, cs0, rho0 = state["reference"]
        # The fifth result, the wavelet gradient, is a point value at the source cell; the tile shape that the
        # operator's timing picks moves its rounding from run to run, so it is not among what is compared.
        J, *grads = fw.compute_misfit(state["fwi"], *state["model"], state["stf"], cp_ref=cp0, cs_ref=cs0,
                                      rho_ref=rho0, with_grad=True)[:4]
        return {"misfit": _single(J), **{k: _single(g) for k, g in zip(("cp", "cs", "rho"), grads)}}
    if call == "inversion":
        J, g, _, illum = state["problem"].misfit_grad(state["vp"], illumination=state["illum"])
        out = {"misfit": _single(J), "vp": _single(g)}
        return out if illum is None else {**out, "illumination": _single(illum)}
    if call == "modelling":
        return state["ctx"].obs(*state["model"], state["stf"], state["ids"], write_files=False)
    if call == "train":
        net = state["net"]
        loss = net.train(state["samples"], 1)
        return {"loss": _single(loss), "W": list(net.W), "b": list(net.b)}
    return _single(state["net"].precondition(*state["args"]))


# ---------------------------------------------------------------------------------------------------------------
# What a call cannot do without.


def _shot_sizes(case):
    rows = case["nz"] + 2 * case["pml"] + _padding(case)
    if not case["aperture"]:
        return [(rows * (case["nx"] + 2 * case["pml"]), case["nt"])] * case["shots"]
    width = (min(case["aperture"], case["nx"]) + case["nx"]) // 2 + 2 * case["pml"]  # the mean of what is drawn
    return [(rows * width, (3 * case["nt"] // 8 + case["nt"]) // 2)] * case["shots"]


def work(case):
    if case["call"] in ("train", "precondition"):
        pixels = case["nz"] * case["nx"]
        macs = 9 * sum(ci * co for ci, co, _, _ in _LAYERS) * pixels
        acts = 2 * sum(ci + co for ci, co, _, _ in _LAYERS) * pixels  # BF16, each layer's input and output
        passes = 3 if case["call"] == "train" else 1
        return {"bytes": passes * acts + 8 * 9 * pixels, "flops": 2 * macs * passes}
    # One time step of one cell, each array in FP32 once: forward, the 5 fields read and written and 5 media; the
    # adjoint, both sets of fields read and written, 5 media and 3 gradients updated. 64 and 200 operations.
    steps = sum(c * n for c, n in _shot_sizes(case))
    adjoint = case["call"] != "modelling"
    traces = sum(n for _, n in _shot_sizes(case)) * case["nx"] * 4
    return {"bytes": steps * (60 + (124 if adjoint else 0)) + traces, "flops": steps * (64 + (200 if adjoint else 0))}


# ---------------------------------------------------------------------------------------------------------------
# The same results in 64 bits: plain torch, the reference's scheme written out.


def _profile(n, length, pml, h, f0, dt):
    """CPML K, a, b at the integer and the half points of an axis of n cells (rows past n: none)."""
    i = torch.arange(n, dtype=torch.float64)
    d0 = -9.0 * 3000.0 * math.log(0.0008) / (2.0 * pml * h)
    out = []
    for half in (0.0, 0.5):
        depth = torch.maximum((pml - i - half) / pml, (pml - n + i + half) / pml)
        x = depth.clamp(min=0.0)
        on = depth >= 0.0
        d = torch.where(on, d0 * (0.25 * x + 0.75 * x ** 8), 0.0)
        k = 1.0 + x ** 8
        al = torch.where(on, (math.pi * f0 * (1.0 - x)).clamp(min=0.0), 0.0)
        b = torch.exp(-(d / k + al) * dt)
        a = torch.where(d.abs() > 1e-6, d * (b - 1.0) / (k * (d + k * al)), 0.0)
        fill = length - n
        out += [torch.cat([v, torch.full((fill,), e, dtype=torch.float64)]) for v, e in ((k, 1.0), (a, 0.0), (b, 1.0))]
    return out


def _taper(nt, dt, ratio, start=None, end=None, weight=None):
    """cos^2-tapered weights of a record, or of each trace with its own window and weight."""
    t = torch.arange(nt, dtype=torch.float64) * dt
    if start is None:
        start, end = torch.zeros(1, dtype=torch.float64), torch.full((1,), nt * dt, dtype=torch.float64)
        weight = torch.ones(1, dtype=torch.float64)
    t0, t3 = (v.clamp(0.0, nt * dt)[:, None] for v in (start, end))
    off = (t3 - t0) * ratio
    t1, t2 = t0 + off, t3 - off
    amp = torch.zeros(len(start), nt, dtype=torch.float64)
    amp = torch.where((t >= t0) & (t < t1), torch.sin(math.pi / 2 * (t - t0) / off), amp)
    amp = torch.where((t >= t1) & (t < t2), torch.ones_like(amp), amp)
    amp = torch.where((t >= t2) & (t < t3), torch.cos(math.pi / 2 * (t - t2) / off), amp)
    return torch.where(off > 0, amp ** 2 * weight[:, None], torch.ones_like(amp))


def _condition(syn, obs, s, case, nt, dt, stf):
    """Residual path of one shot: (sum of squares, adjoint source, wavelet the reverse pass subtracts)."""
    dev = syn.device
    if case["windows"]:
        win = [torch.tensor(s[k], dtype=torch.float64) for k in ("win_start", "win_end", "weights")]
        w_obs, w_res = (_taper(nt, dt, r, *win).to(dev) for r in (0.005, 0.1))
    else:
        w_obs = w_res = _taper(nt, dt, 0.005).to(dev)
    syn, obs = syn * w_obs, obs * w_obs

    def spectral(x, gain):
        return torch.fft.irfft(torch.fft.rfft(x, 2 * nt) * gain, 2 * nt)[..., :nt]

    band = None
    if case["band"]:
        f = torch.arange(nt + 1, dtype=torch.float64, device=dev) / (2 * nt * dt)
        c0, c1, c2, c3 = _corners(case)
        band = torch.zeros_like(f)
        band = torch.where((f >= c0) & (f < c1), torch.sin(math.pi / 2 * (f - c0) / (c1 - c0)), band)
        band = torch.where((f >= c1) & (f < c2), torch.ones_like(f), band)
        band = torch.where((f >= c2) & (f < c3), torch.cos(math.pi / 2 * (f - c2) / (c3 - c2)), band) ** 2
        syn, obs = spectral(syn, band), spectral(obs, band)
    coef = None
    if case["update"]:
        w2 = _taper(2 * nt, dt, 0.01)[:, :nt].to(dev)
        O, C = torch.fft.rfft(obs * w2, 2 * nt), torch.fft.rfft(syn * w2, 2 * nt)
        coef = (C.conj() * O).sum(0) / ((C.abs() ** 2).sum(0) + 1e-6)
        syn, stf = spectral(syn * w2, coef), spectral(stf, coef)
    res = obs - syn
    res[:, 0] = 0.0
    total = (res ** 2).sum()
    if coef is not None:
        res = spectral(res * w2, coef)
    if band is not None:
        res = spectral(res, band)
    return total, res * w_res, stf


def _simulate(case, w, members, adjoint, device):
    """The shots `members` (same sub-grid width and record) together. Returns (misfit, gathers, gradients w.r.t.
    lambda, mu [MPa], rho and the wavelets, illumination), on the shots' own columns."""
    T = dict(dtype=torch.float64, device=device)
    pml, pad, dt, h = case["pml"], w["pad"], w["dt"], case["dx"]
    shots = [w["shots"][k] for k in members]
    S, nt = len(shots), shots[0].get("nSteps", case["nt"])
    nz = w["vp"].shape[0]
    nx = shots[0]["win_x1"] - shots[0]["win_x0"] + 1 + 2 * pml if case["aperture"] else w["vp"].shape[1]
    cols = [s.get("win_x0", 0) for s in shots]
    lam, mu, rho = (torch.stack([torch.from_numpy(w[k][:, c:c + nx] * f) for c in cols]).to(device)
                    for k, f in (("lam", 1e6), ("mu", 1e6), ("rho", 1.0)))
    # The package stores the moduli and the density in FP32: its input precision.
    lam, mu, rho = (v.float().double() for v in (lam, mu, rho))
    ave = torch.zeros_like(mu)
    bA, bB = torch.full_like(rho, 1e-3), torch.full_like(rho, 1e-3)
    core = (slice(None), slice(2, nz - 2), slice(2, nx - 2))
    nxt = lambda v, a, b: v[:, 2 + a:nz - 2 + a, 2 + b:nx - 2 + b]  # noqa: E731
    ave[core] = 4.0 / (1 / nxt(mu, 0, 0) + 1 / nxt(mu, 1, 0) + 1 / nxt(mu, 0, 1) + 1 / nxt(mu, 1, 1))
    bA[core] = 2.0 / (nxt(rho, 1, 0) + nxt(rho, 0, 0))
    bB[core] = 2.0 / (nxt(rho, 0, 1) + nxt(rho, 0, 0))
    # A windowed shot's averages come from the full model, also at the edge columns of its sub-grid.
    for k, c in enumerate(cols):
        if c > 0 or c + nx < w["vp"].shape[1]:
            full = torch.from_numpy(w["mu"] * 1e6).to(device).float().double()
            den = torch.from_numpy(w["rho"]).to(device).float().double()
            a, e, f = torch.zeros_like(full), torch.full_like(full, 1e-3), torch.full_like(full, 1e-3)
            i = (slice(2, -2), slice(2, -2))
            a[i] = 4.0 / (1 / full[2:-2, 2:-2] + 1 / full[3:-1, 2:-2] + 1 / full[2:-2, 3:-1] + 1 / full[3:-1, 3:-1])
            e[i] = 2.0 / (den[3:-1, 2:-2] + den[2:-2, 2:-2])
            f[i] = 2.0 / (den[2:-2, 3:-1] + den[2:-2, 2:-2])
            ave[k], bA[k], bB[k] = a[:, c:c + nx], e[:, c:c + nx], f[:, c:c + nx]
    dom = (slice(None), slice(2, nz - pad - 2), slice(2, nx - 2))
    D = lambda v: v[dom]  # noqa: E731
    sh = lambda v, a, b: v[:, 2 + a:nz - pad - 2 + a, 2 + b:nx - 2 + b]  # noqa: E731
    C1, C2 = 1.125, 1.0 / 24.0
    dmz = lambda v: (C1 * (sh(v, 0, 0) - sh(v, -1, 0)) - C2 * (sh(v, 1, 0) - sh(v, -2, 0))) / h  # noqa: E731
    dpz = lambda v: (C1 * (sh(v, 1, 0) - sh(v, 0, 0)) - C2 * (sh(v, 2, 0) - sh(v, -1, 0))) / h  # noqa: E731
    dmx = lambda v: (C1 * (sh(v, 0, 0) - sh(v, 0, -1)) - C2 * (sh(v, 0, 1) - sh(v, 0, -2))) / h  # noqa: E731
    dpx = lambda v: (C1 * (sh(v, 0, 1) - sh(v, 0, 0)) - C2 * (sh(v, 0, 2) - sh(v, 0, -1))) / h  # noqa: E731
    f0 = _f0(case)
    Kz, az, bz, Kzh, azh, bzh = (v.to(device)[2:nz - pad - 2, None] for v in _profile(nz - pad, nz, pml, h, f0, dt))
    Kx, ax, bx, Kxh, axh, bxh = (v.to(device)[None, 2:nx - 2] for v in _profile(nx, nx, pml, h, f0, dt))
    x = torch.arange(2, nx - 2, device=device)[None, :]
    z = torch.arange(2, nz - pad - 2, device=device)[:, None]
    zp = (z < pml) | (z > nz - pml - pad - 1)
    xp = (x < pml) | (x > nx - pml - 1)
    xv = (x < pml) | (x > nx - pml)  # the forward velocity's own layer starts a column later
    one, zero = torch.ones_like(Kx), torch.zeros_like(Kx)
    Kxv, axv, Kxhv, axhv = (torch.where(xv, a, b) for a, b in ((Kx, one), (ax, zero), (Kxh, one), (axh, zero)))
    l2m = lam + 2.0 * mu
    lamD, l2mD, aveD, bAD, bBD = D(lam), D(l2m), D(ave), D(bA), D(bB)
    new = lambda: torch.zeros(S, nz, nx, **T)  # noqa: E731
    vz, vx, szz, sxx, sxz = (new() for _ in range(5))
    mem = [torch.zeros_like(lamD) for _ in range(8)]
    taper = _taper(nt, dt, 0.001)[0]
    stf = torch.stack([torch.from_numpy(w["stf"][k][:nt]).float().double() * taper for k in members]).to(device)
    at = torch.arange(S, device=device)
    sz = torch.tensor([s["z_src"] + pml for s in shots], device=device)
    sx = torch.tensor([s["x_src"] + pml - c for s, c in zip(shots, cols)], device=device)
    rz = [torch.tensor(s["z_rec"], device=device) + pml for s in shots]
    rx = [torch.tensor(s["x_rec"], device=device) + pml - c for s, c in zip(shots, cols)]
    rs = torch.cat([torch.full_like(v, k) for k, v in enumerate(rz)])
    rz, rx, nrec = torch.cat(rz), torch.cat(rx), [len(v) for v in rz]
    ring = torch.zeros(nz, nx, dtype=torch.bool)
    ring[pml - 2:nz - pml - pad + 2, pml - 2:nx - pml + 2] = True
    ring[pml + 3:nz - pml - pad - 3, pml + 3:nx - pml - 3] = False
    ring = ring.reshape(-1).nonzero()[:, 0].to(device)
    flat = lambda v: v.reshape(S, nz * nx)  # noqa: E731
    store = torch.empty(nt - 1, 5, S, len(ring), **T) if adjoint else None
    data = torch.zeros(len(rs), nt, **T)
    illum = new() if case["illum"] else None
    scale = 2250000.0

    def pml_step(k, b, a, K, d):
        mem[k].mul_(b).add_(a * d)
        return d / K + mem[k]

    for it in range(nt - 1):
        if adjoint:
            for q, v in enumerate((szz, sxz, sxx, vz, vx)):
                torch.index_select(flat(v), 1, ring, out=store[it, q])
        a = pml_step(0, bz, torch.where(zp, az, 0.0), torch.where(zp, Kz, 1.0), dmz(vz))
        b = pml_step(1, bzh, torch.where(zp, azh, 0.0), torch.where(zp, Kzh, 1.0), dpz(vx))
        c = pml_step(2, bx, torch.where(xp, ax, 0.0), torch.where(xp, Kx, 1.0), dmx(vx))
        d = pml_step(3, bxh, torch.where(xp, axh, 0.0), torch.where(xp, Kxh, 1.0), dpx(vz))
        D(szz).add_((l2mD * a + lamD * c) * dt)
        D(sxx).add_((lamD * a + l2mD * c) * dt)
        D(sxz).add_(aveD * (b + d) * dt)
        szz[at, sz, sx] += scale * dt * stf[:, it]
        sxx[at, sz, sx] += 3.0 * scale * dt * stf[:, it]
        data[:, it + 1] = szz[rs, rz, rx] + 3.0 * sxx[rs, rz, rx]
        a = pml_step(4, bzh, torch.where(zp, azh, 0.0), torch.where(zp, Kzh, 1.0), dpz(szz))
        b = pml_step(5, bx, axv, Kxv, dmx(sxz))
        c = pml_step(6, bz, torch.where(zp, az, 0.0), torch.where(zp, Kz, 1.0), dmz(sxz))
        d = pml_step(7, bxh, axhv, Kxhv, dpx(sxx))
        D(vz).add_((a + b) * bAD * dt)
        D(vx).add_((c + d) * bBD * dt)
        if illum is not None:
            D(illum).add_(D(vz) ** 2 + D(vx) ** 2)
    gathers = list(torch.split(data, nrec))
    if not adjoint:
        return None, gathers, None, None, illum
    total, res, back = 0.0, [], []
    for k, (s, g) in enumerate(zip(shots, gathers)):
        o = torch.from_numpy(w["obs"][members[k]]).to(device).double()
        j, r, b = _condition(g, o, s, case, nt, dt, stf[k])
        total, res, back = total + 0.5 * j, res + [r], back + [b]
    res, back = torch.cat(res), torch.stack(back)

    za, xa, pzz, pxx, pxz = (new() for _ in range(5))  # adjoint velocities and stresses
    psi = [new() for _ in range(8)]  # of dvz_dz, dvz_dx, dvx_dz, dvx_dx, dszz_dz, dsxx_dx, dsxz_dz, dsxz_dx
    inner = (slice(None), slice(pml - 2, nz - pad - pml - 2), slice(pml - 2, nx - pml - 2))  # interior in domain arrays
    I = (slice(None), slice(pml, nz - pad - pml), slice(pml, nx - pml))  # noqa: E741
    gl, gm, tau, ta, tb = (torch.zeros_like(lam[I]) for _ in range(5))
    g_stf = torch.zeros(S, nt, **T)

    def inject_and_stress(it):
        pzz.index_put_((rs, rz, rx), res[:, it], accumulate=True)
        pxx.index_put_((rs, rz, rx), 3.0 * res[:, it], accumulate=True)
        D(pxz).add_((-dpx(za) / Kx * bAD - dpz(xa) / Kz * bBD) * dt - ax * dpx(psi[7]) - az * dpz(psi[6]))
        step = D(pxz) * aveD * dt
        D(psi[1]).mul_(bxh).add_(step)
        D(psi[2]).mul_(bzh).add_(step)
        tx = -bBD * dmx(xa) / Kxh * dt - axh * dmx(psi[5])
        tz = -bAD * dmz(za) / Kzh * dt - azh * dmz(psi[4])
        D(pxx).add_(tx)
        D(pzz).add_(tz)
        D(psi[3]).mul_(bx).add_((lamD * D(pzz) + l2mD * D(pxx)) * dt)
        D(psi[0]).mul_(bz).add_((l2mD * D(pzz) + lamD * D(pxx)) * dt)

    def reverse_velocity(it):
        g_stf[:, it] = -(pzz[at, sz, sx] + 3.0 * pxx[at, sz, sx]) * dt
        ea, eb = (dpz(szz) + dmx(sxz))[inner], (dmz(sxz) + dpx(sxx))[inner]
        vz[I].sub_(ea * bA[I] * dt)
        vx[I].sub_(eb * bB[I] * dt)
        ta.add_(za[I] * ea)
        tb.add_(xa[I] * eb)
        flat(vz)[:, ring] = store[it, 3]
        flat(vx)[:, ring] = store[it, 4]

    def reverse_stress(it):
        szz[at, sz, sx] -= scale * dt * back[:, it]
        sxx[at, sz, sx] -= 3.0 * scale * dt * back[:, it]
        a, c, e = dmz(vz)[inner], dmx(vx)[inner], (dpz(vx) + dpx(vz))[inner]
        szz[I].sub_((l2m[I] * a + lam[I] * c) * dt)
        sxx[I].sub_((lam[I] * a + l2m[I] * c) * dt)
        sxz[I].sub_(ave[I] * e * dt)
        gl.sub_((pzz[I] + pxx[I]) * (a + c))
        gm.sub_(2.0 * (pzz[I] * a + pxx[I] * c))
        tau.sub_(pxz[I] * e)
        for q, v in enumerate((szz, sxz, sxx)):
            flat(v)[:, ring] = store[it, q]

    def velocity(it):
        D(xa).add_((-(lamD * dpx(pzz) + l2mD * dpx(pxx)) / Kx - aveD / Kzh * dmz(pxz)) * dt - ax * dpx(psi[3])
                   - azh * dmz(psi[2]))
        step = bBD * D(xa) * dt
        D(psi[5]).copy_(torch.where(xp, bxh * D(psi[5]) + step, D(psi[5])))
        D(psi[6]).copy_(torch.where(zp, bz * D(psi[6]) + step, D(psi[6])))
        D(za).add_((-(l2mD * dpz(pzz) + lamD * dpz(pxx)) / Kz - aveD / Kxh * dmx(pxz)) * dt - az * dpz(psi[0])
                   - axh * dmx(psi[1]))
        step = bAD * D(za) * dt
        D(psi[7]).copy_(torch.where(xp, bx * D(psi[7]) + step, D(psi[7])))
        D(psi[4]).copy_(torch.where(zp, bzh * D(psi[4]) + step, D(psi[4])))

    inject_and_stress(nt - 1)
    for it in range(nt - 2, -1, -1):
        reverse_velocity(it)
        reverse_stress(it)
        velocity(it)
        inject_and_stress(it)
    # The chain rules of the averaged shear modulus and of the buoyancies, applied to the sums over time.
    g = [new() for _ in range(3)]
    g[0][I] = gl * dt * 1e6
    g[1][I] = gm * dt * 1e6
    h2 = (ave ** 2 / 4.0)[I] * tau * dt * 1e6
    w2, (zs, xs) = 1.0 / mu ** 2, (I[1], I[2])
    wide = torch.zeros(S, h2.shape[1], h2.shape[2] + 1, **T)  # columns xi0 .. xi1 + 1
    own = torch.cat([h2, torch.zeros_like(h2[:, :, :1])], 2)
    left = torch.cat([torch.zeros_like(h2[:, :, :1]), h2], 2)
    wide += own + left
    wide[:, 1:] += own[:, :-1]
    wide[:, 1:, :-1] += left[:, :-1, :-1]
    g[1][:, zs, xs.start:xs.stop + 1] += w2[:, zs, xs.start:xs.stop + 1] * wide
    ta, tb = ta * bA[I] ** 2 * dt / 2.0, tb * bB[I] ** 2 * dt / 2.0
    wide = torch.zeros_like(wide)
    wide[:, :, :-1] += ta + tb
    wide[:, 1:, :-1] += ta[:, :-1]
    wide[:, :, 1:] += tb
    g[2][:, zs, xs.start:xs.stop + 1] += wide
    return total, gathers, g, g_stf, illum


def _exact_fwi(case, seed):
    adjoint = case["call"] != "modelling"
    w = _world(case, seed)
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if case["call"] == "misfit" or case["call"] == "inversion":
        m = _mask(case, w["pad"])
        vp0 = _start_vp(case, w["vp"])
        if case["call"] == "misfit":
            full = {"cp": w["vp"] * m + vp0 * (1 - m), "cs": w["vs"] * m + vp0 / math.sqrt(3.0) * (1 - m),
                    "rho": w["rho"] * m + 310.0 * vp0 ** 0.25 * (1 - m)}
        else:
            v = np.clip(vp0 * (1 - m) + w["vp"] * m, 1400.0, 5000.0)
            full = {"cp": v, "cs": v / math.sqrt(3.0), "rho": 310.0 * v ** 0.25}
        w["lam"] = (full["cp"] ** 2 - 2.0 * full["cs"] ** 2) * full["rho"] / 1e6
        w["mu"], w["rho"] = full["cs"] ** 2 * full["rho"] / 1e6, full["rho"]
    alike = {}
    for k, s in enumerate(w["shots"]):
        alike.setdefault((len(s["x_rec"]) if case["aperture"] else 0, s.get("nSteps", 0)), []).append(k)
    # About 1.5 ms of launches a step, and 130 passes over a field of a group's shots in double.
    cells = {k: len(v) * w["vp"].shape[0] * (k[0] + 2 * case["pml"] if k[0] else w["vp"].shape[1])
             for k, v in alike.items()}
    seconds = sum((k[1] or case["nt"]) * ((2.2e-3 if adjoint else 0.7e-3) + cells[k] * 8 * (400 if adjoint else 120) / 5e12)
                  for k in alike)
    stored = max((k[1] or case["nt"]) * 5 * 8 * len(v) * 10 * sum(w["vp"].shape) for k, v in alike.items())
    if seconds > 18 or stored > 60e9:
        return None
    total, gathers = 0.0, [None] * case["shots"]
    nz, nx = w["vp"].shape
    g = [np.zeros((nz, nx)) for _ in range(3)]
    illum = np.zeros((nz, nx)) if case["illum"] else None
    g_stf = np.zeros((case["shots"], case["nt"]))
    for key, members in alike.items():
        j, data, grads, gs, ill = _simulate(case, w, members, adjoint, device)
        for k, d in zip(members, data):
            gathers[k] = d
        if not adjoint:
            continue
        total += float(j)
        for q, k in enumerate(members):
            c = w["shots"][k].get("win_x0", 0)
            for a, b in zip(g, grads):
                a[:, c:c + b.shape[2]] += b[q].cpu().numpy()
            g_stf[k, :gs.shape[1]] = gs[q].cpu().numpy()
            if illum is not None:
                illum[:, c:c + ill.shape[2]] += ill[q].cpu().numpy()
    if not adjoint:
        return gathers
    gl, gm, gd = g
    if case["call"] == "gradient":
        return {"misfit": np.float64(total), "lam": gl, "mu": gm, "den": gd, "stf": g_stf}
    cp, cs, rho = full["cp"], full["cs"], full["rho"]
    if case["call"] == "misfit":
        return {"misfit": np.float64(total), "cp": gl * 2 * cp * rho / 1e6 * m,
                "cs": (gl * (-4 * cs) + gm * 2 * cs) * rho / 1e6 * m,
                "rho": (gd + gl * (cp ** 2 - 2 * cs ** 2) / 1e6 + gm * cs ** 2 / 1e6) * m}
    drho = 77.5 * cp ** -0.75
    out = {"misfit": np.float64(total), "vp": ((gl + gm) * (drho * cp * cp + 2.0 * rho * cp) / 3e6 + gd * drho) * m}
    return out if illum is None else {**out, "illumination": illum}


def _exact_net(case, seed):
    grads, illum, mask, weights = _net_inputs(case, seed)
    feats, e = _features(grads, illum, mask)
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    x = torch.from_numpy(feats).to(device)[None]
    for k, (ci, co, _, _) in enumerate(_LAYERS):
        wk = torch.from_numpy(weights[f"W{k}"]).double().to(device)[:, :ci, :co].reshape(3, 3, ci, co)
        x = torch.nn.functional.pad(x, (1, 1, 1, 1))
        y = torch.from_numpy(weights[f"b{k}"]).double().to(device)[:co, None, None].expand(co, case["nz"], case["nx"])
        y = y.clone()
        for a in range(3):
            for b in range(3):
                y += torch.einsum("io,izx->ozx", wk[a, b], x[0, :, a:a + case["nz"], b:b + case["nx"]])
        x = (0.5 * y * (1.0 + torch.erf(y / math.sqrt(2.0))) if k < 5 else y)[None]
    out = x[0].cpu().numpy()
    if case["call"] == "precondition":
        return np.stack(grads) * np.exp(np.clip(out, -30.0, 5.0)) * mask
    target = np.log(1e-3 / (e + 1e-3)) * mask
    loss = np.sum(((out - target) * mask) ** 2) / (3.0 * mask.sum())
    # The weights after a step have no such value: the optimiser's first step is the sign of the gradient, and BF16
    # activations decide the signs of the smallest.
    return {"loss": np.array([loss]), "W": [None] * 6, "b": [None] * 6}


def exact(case, seed):
    if case["call"] in ("train", "precondition"):
        return _exact_net(case, seed)
    return _exact_fwi(case, seed)
