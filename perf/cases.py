"""The work this engine is used for, as measurable cases.

Four kinds, each through the Python package's public calls:

  synth    gm_synthesize: Stokes profiles of given models, with or without
           their response functions
  invert   gm_invert / gm_invert_ex: one cube on one grid, in device or host
           memory, from the classical or the learned start
  rois     gm_invert_rois: regions of interest on many grids in one call
  predict  gm_mlp_predict: start models from a network
  train    gm_mlp_train: a network fitted to synthesised profiles

The line is Fe I 6173.3356 A; truth models, noise, PSF, stray light, guess
model and iteration limit are those of bench.py and tests/helpers.py.
Observations are formed in float64 torch by the functions below, so that they
depend on the seed alone.
"""
import ctypes
import gc
import json
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "g-milos_b200") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "g-milos_b200"))
import gmilos_b200 as G  # noqa: E402

LAMBDA0 = 6173.3356
VLIGHT = 2.99792458e5
LARMOR = 4.6686411e-13
NOISE = 1e-3
FWHM_MA = 100.0
MAXITER = 50
GUESS = (40.0, 1000.0, 0.2, 0.03, 0.05, 150.0, 110.0, 0.35, 0.5, 0.0, 1.0)
GUESS_VMAC = GUESS[:9] + (0.5, 1.0)
STRAY_MODEL = (10.0, 0.0, 0.0, 0.03, 0.1, 0.0, 0.0, 0.3, 0.7, 0.0, 1.0)
FIX = {"nine": (1,) * 9 + (0, 0),              # the 9 Milne-Eddington parameters
       "seven": (1,) * 7 + (0, 0, 0, 1),       # S0, S1 fixed, filling factor free
       "ten": (1,) * 9 + (0, 1),               # and the filling factor
       "eleven": (1,) * 11}                    # and v_mac: the 11-term path


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # interactive synthesis of one model with its response functions (the
        # reference's kernel_synthesis call): latency
        {"name": "synth_one_rf", "kind": "synth", "pixels": 1, "nl": 30, "psf": True, "rf": True, "stray": False,
         "f64": True},
        # response functions of an ordinary field of view (sensitivity studies)
        {"name": "synth_map_rf", "kind": "synth", "pixels": 20000, "nl": 30, "psf": True, "rf": True, "stray": True,
         "f64": True},
        # profiles only: a training set for the learned guess
        {"name": "synth_training_set", "kind": "synth", "pixels": 262144, "nl": 30, "psf": True, "rf": False,
         "stray": False, "f64": True},
        # the reference's CPU-runnable example: a small cube without PSF
        {"name": "invert_64x64", "kind": "invert", "pixels": 4096, "nl": 30, "psf": False, "stray": False,
         "free": "nine", "start": "classical", "stop": 0.0, "numerics": 0, "host": False},
        # a ragged-sized cut-out with everything modelled
        {"name": "invert_37x53", "kind": "invert", "pixels": 1961, "nl": 30, "psf": True, "stray": True,
         "free": "ten", "start": "classical", "stop": 0.0, "numerics": 0, "host": False},
        # the headline cube, resident on the device
        {"name": "invert_cube", "kind": "invert", "pixels": 1 << 20, "nl": 30, "psf": True, "stray": True,
         "free": "ten", "start": "classical", "stop": 0.0, "numerics": 0, "host": False},
        # a finely sampled line: two samples per lane
        {"name": "invert_45_samples", "kind": "invert", "pixels": 170 * 170, "nl": 45, "psf": True, "stray": False,
         "free": "nine", "start": "classical", "stop": 0.0, "numerics": 0, "host": False},
        # v_mac and the filling factor free: the FP64 11-term path
        {"name": "invert_vmac_free", "kind": "invert", "pixels": 96 * 96, "nl": 30, "psf": True, "stray": True,
         "free": "eleven", "start": "classical", "stop": 0.0, "numerics": 0, "host": False},
        # a cube in host memory, learned start, early stop: the pipelined path end to end
        {"name": "invert_host_learned", "kind": "invert", "pixels": 520 * 520, "nl": 30, "psf": True, "stray": False,
         "free": "nine", "start": "learned", "stop": 1e-4, "numerics": 0, "host": True},
        # a dozen regions on their own grids, early stop
        {"name": "rois_12", "kind": "rois", "rois": 12, "side_min": 16, "side_max": 160, "nl_min": 12, "nl_max": 60,
         "psf": False, "stop": 1e-4, "layout": 3},
        # start models of a cube
        {"name": "predict_cube", "kind": "predict", "pixels": (1 << 18) + 77, "nl": 30, "host": False},
        # a network trained on a modest set
        {"name": "train_128k", "kind": "train", "pixels": 1 << 17, "nl": 30, "epochs": 2, "batch": 8192},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["synth", "synth", "invert", "invert", "invert", "rois", "predict", "train"])
    if kind == "synth":
        rf = rng.random() < 0.5
        return {"kind": kind, "pixels": _log(rng, 1, 40000 if rf else 400000), "nl": rng.randint(8, 64),
                "psf": rng.random() < 0.7, "rf": rf, "stray": rng.random() < 0.4, "f64": rng.random() < 0.7}
    if kind == "invert":
        free = rng.choice(["nine", "nine", "ten", "ten", "seven", "eleven"])
        # 14 samples leave degrees of freedom for every parameter; the network reads up to 32
        start = "learned" if rng.random() < 0.2 and free != "eleven" else "classical"
        return {"kind": kind, "pixels": _log(rng, 1, 131072), "nl": rng.randint(14, 32 if start == "learned" else 60),
                "psf": rng.random() < 0.6, "stray": free in ("ten", "seven", "eleven"), "free": free, "start": start,
                "stop": rng.choice([0.0, 1e-4]), "numerics": rng.choice([0, 0, 0, 1]), "host": rng.random() < 0.3}
    if kind == "rois":
        a = rng.randint(4, 40)
        return {"kind": kind, "rois": rng.randint(2, 14), "side_min": a, "side_max": a + rng.randint(8, 120),
                "nl_min": rng.randint(12, 30), "nl_max": rng.randint(31, 60), "psf": rng.random() < 0.5,
                "stop": rng.choice([0.0, 1e-4]), "layout": rng.randint(0, 1 << 20)}
    if kind == "predict":
        return {"kind": kind, "pixels": _log(rng, 1, 1 << 20), "nl": rng.randint(8, 32), "host": rng.random() < 0.3}
    return {"kind": kind, "pixels": _log(rng, 1 << 14, 1 << 18), "nl": rng.randint(12, 32), "epochs": rng.randint(1, 2),
            "batch": 128 * _log(rng, 16, 128)}


# ---------------------------------------------------------------- inputs
def _grid(nl):
    """nl samples of 35 mA; 30 samples are the -350:35:665 grid, others are centred."""
    return (-350.0 + 35.0 * np.arange(nl) if nl == 30 else 35.0 * (np.arange(nl) - nl // 2)) / 1000.0


def _truth(n, g, alpha=False):
    r = torch.rand((n, 11), generator=g, device="cuda", dtype=torch.float64)
    lo = torch.tensor([1, 0, -3, 0.020, 0, 0, 0, 0.1, 0.3, 0, 0.7], dtype=torch.float64, device="cuda")
    hi = torch.tensor([30, 3000, 3, 0.060, 0.5, 180, 180, 0.5, 1.0, 0, 1.0], dtype=torch.float64, device="cuda")
    t = lo + (hi - lo) * r
    t[:, 7:9] /= t[:, 7:9].sum(dim=1, keepdim=True)
    if not alpha:
        t[:, 10] = 1.0
    return t


def _voigt(a, v):
    """Voigt and Faraday-Voigt functions by the rational approximation of Hui, Armstrong & Wray (1978)."""
    p = (122.607931777104326, 214.382388694706425, 181.928533092181549, 93.155580458138441, 30.180142196210589,
         5.912626209773153, 0.564189583562615)
    q = (122.60793177387535, 352.730625110963558, 457.334478783897737, 348.703917719495792, 170.354001821091472,
         53.992906912940207, 10.479857114260399)
    z = torch.complex(a.expand_as(v), -v)
    num = torch.full_like(z, p[6])
    for c in p[5::-1]:
        num = num * z + c
    den = torch.ones_like(z)
    for c in q[6::-1]:
        den = den * z + c
    w = num / den
    return w.real, w.imag * 0.5


def _zeeman():
    z = G.fe6173()[1]
    pi = [(z.nup[i], z.wep[i]) for i in range(z.n_pi)]
    blue = [(z.nub[i], z.web[i]) for i in range(z.n_sig)]
    red = [(-z.nub[z.n_sig - 1 - i], z.wer[i]) for i in range(z.n_sig)]
    return (pi, blue, red), z.fo


def _correlate(x, taps, reflect):
    """Same-size correlation of the last axis with the taps centred at nl / 2, zero padded;
    reflected about max(first, last) where asked."""
    nl = x.shape[-1]
    k = torch.arange(nl, device=x.device)
    j = k[:, None] - k[None, :] + nl // 2
    h = torch.as_tensor(taps, dtype=torch.float64, device=x.device)
    T = torch.where((j >= 0) & (j < nl), h[j.clamp(0, nl - 1)], torch.zeros((), dtype=torch.float64, device=x.device))
    if not reflect:
        return x @ T
    ic = torch.maximum(x[..., :1], x[..., -1:])
    return ic - (ic - x) @ T


def _profiles(m, off, taps=None, stray=None, rf=False):
    """Stokes profiles [P][4][nl] of the models in float64, and their response functions
    [P][4][10][nl] (analytic; the last slot is the filling factor's; as in the reference,
    me_der.cu:53-77, the dispersion profile's derivative is that of the Faraday-Voigt function
    alone, without the profile's factor 2)."""
    groups, fo = _zeeman()
    P, nl = m.shape[0], len(off)
    o = torch.as_tensor(off, dtype=torch.float64, device=m.device)[None]
    col = lambda i: m[:, i:i + 1]  # noqa: E731
    rad = math.pi / 180.0
    cg, sg = torch.cos(col(5) * rad), torch.sin(col(5) * rad)
    ca, sa = torch.cos(2 * col(6) * rad), torch.sin(2 * col(6) * rad)
    e2 = col(0) * fo / 2
    dopp, damp = col(3), col(4)
    shift = LAMBDA0 * LAMBDA0 / dopp * LARMOR
    base = o / dopp - col(2) * LAMBDA0 / (VLIGHT * dopp)
    fi, fs, dfi, dfs = [], [], [], []
    for comps in groups:
        a = s = 0
        da, ds = [0, 0, 0, 0], [0, 0, 0, 0]
        for nu, w in comps:
            v = base - shift * nu * col(1)
            h, f = _voigt(damp, v)
            a, s = a + w * h, s + 2 * w * f
            if rf:
                dh, df = w * (4 * damp * f - 2 * v * h), w * (1 / math.sqrt(math.pi) - damp * h - 2 * v * f)
                dv = (-shift * nu, -LAMBDA0 / (VLIGHT * dopp), -v / dopp)
                for k in range(3):
                    da[k], ds[k] = da[k] + dh * dv[k], ds[k] + df * dv[k]
                da[3], ds[3] = da[3] - 2 * df, ds[3] + dh / 2
        fi.append(a)
        fs.append(s)
        dfi.append(da)
        dfs.append(ds)

    def matrix(f, e2, cg, sg, ca, sa):
        lin = e2 * (f[0] - (f[1] + f[2]) / 2) * sg * sg
        return (e2 * (f[0] * sg * sg + (f[1] + f[2]) * (1 + cg * cg) / 2), lin * ca, lin * sa, e2 * (f[2] - f[1]) * cg)

    ei, eq, eu, ev = matrix(fi, e2, cg, sg, ca, sa)
    _, rq, ru, rv = matrix(fs, e2, cg, sg, ca, sa)
    ei = 1 + ei
    s1 = col(8)

    def solve(ei, eq, eu, ev, rq, ru, rv):
        g = eq * rq + eu * ru + ev * rv
        r2 = rq * rq + ru * ru + rv * rv
        det = ei * ei * (ei * ei - eq * eq - eu * eu - ev * ev + r2) - g * g
        return (ei * (ei * ei + r2) / det, -(ei * ei * eq + ei * (ev * ru - eu * rv) + rq * g) / det,
                -(ei * ei * eu + ei * (eq * rv - ev * rq) + ru * g) / det,
                -(ei * ei * ev + ei * (eu * rq - eq * ru) + rv * g) / det)

    args = (ei, eq, eu, ev, rq, ru, rv)
    x = solve(*args)
    pure = torch.stack([col(7) + s1 * x[0]] + [s1 * k for k in x[1:]], dim=1)
    grads = []
    if rf:
        # directions of the absorption and dispersion terms per parameter
        dirs = [[t / col(0) for t in (ei - 1, eq, eu, ev, rq, ru, rv)]]
        for k in range(4):
            d = matrix([dfi[j][k] for j in range(3)], e2, cg, sg, ca, sa)
            r = matrix([dfs[j][k] for j in range(3)], e2, cg, sg, ca, sa)
            dirs.append(list(d) + list(r[1:]))
        lin, lins = e2 * (fi[0] - (fi[1] + fi[2]) / 2), e2 * (fs[0] - (fs[1] + fs[2]) / 2)
        d2 = 2 * sg * cg * rad
        dirs.append([e2 * (fi[0] - (fi[1] + fi[2]) / 2) * d2, lin * d2 * ca, lin * d2 * sa, -e2 * (fi[2] - fi[1]) * sg * rad,
                     lins * d2 * ca, lins * d2 * sa, -e2 * (fs[2] - fs[1]) * sg * rad])
        zero = torch.zeros_like(ei)
        dirs.append([zero, -2 * rad * eu, 2 * rad * eq, zero, -2 * rad * ru, 2 * rad * rq, zero])
        for d in dirs:
            grads.append(s1[:, None] * torch.stack(torch.func.jvp(solve, args, tuple(d))[1], dim=1))
        one = torch.zeros_like(pure)
        one[:, 0] = 1.0
        grads += [one, torch.stack(x, dim=1)]
    if taps is not None:
        conv = lambda y: torch.cat([_correlate(y[:, :1], taps, True), _correlate(y[:, 1:], taps, False)], dim=1)  # noqa: E731
        pure = conv(pure)
        grads = [g if i == 7 else conv(g) for i, g in enumerate(grads)]
    mixed, alpha = pure, m[:, 10][:, None, None]
    da = torch.zeros_like(pure)
    if stray is not None:
        sl = torch.as_tensor(stray, dtype=torch.float64, device=m.device)[None]
        mixed, da = alpha * pure + (1 - alpha) * sl, pure - sl
        grads = [alpha * g for g in grads]
    return (mixed, torch.stack(grads + [da], dim=2)) if rf else mixed


def _observe(truth, off, taps, stray, g, noise=NOISE):
    out = torch.empty((truth.shape[0], 4, len(off)), dtype=torch.float32, device="cuda")
    for a in range(0, truth.shape[0], 65536):
        out[a:a + 65536] = _profiles(truth[a:a + 65536], off, taps, stray)
    return out.add_(noise * torch.randn(out.shape, generator=g, device="cuda", dtype=torch.float32))


def _taps(off, psf):
    return G.psf_gaussian(FWHM_MA, LAMBDA0 + off) if psf else None


def _stray(off, taps):
    m = torch.tensor([STRAY_MODEL], dtype=torch.float64, device="cuda")
    return _profiles(m, off, taps)[0].float().cpu().numpy()


def _network(nl):
    """A network with random weights whose outputs land inside the parameters' ranges."""
    net = G.mlp_new(nl, 11 + nl)
    a = net.arrays()
    r = np.random.default_rng(nl)
    a["b1"][:] = r.normal(0, 0.1, a["b1"].shape)
    a["b2"][:] = r.normal(0, 0.1, a["b2"].shape)
    a["w3"][:] *= 10.0
    a["b3"][:9] = r.normal(0, 0.1, 9)
    a["out_mean"][:9] = (15.5, 0, 0.04, 0.25, 0.32, 0.68, 0, 0, 0)
    a["out_scale"][:9] = (8.0, 1.7, 0.011, 0.14, 0.13, 0.13, 700, 700, 700)
    a["in_mean"][:nl] = 0.85
    a["in_scale"][:4 * nl] = np.repeat((6.0, 15.0, 15.0, 10.0), nl)
    return net


# One engine, kept by a program for all its inputs of one configuration.
_kept = {}


def _engine(case):
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    if key not in _kept:
        for e in _kept.values():
            e[0].close()
        _kept.clear()
        gc.collect()
        torch.cuda.empty_cache()
        eng = G.Engine(0)
        net = None
        kind = case["kind"]
        off = _grid(case.get("nl", 30))
        taps = _taps(off, case.get("psf", False) and kind != "rois")
        stray = _stray(off, taps) if case.get("stray") else None
        kw = {"fix": FIX["nine"], "init": GUESS, "miter": MAXITER}
        if kind == "invert":
            kw["fix"] = FIX[case["free"]]
            kw["init"] = GUESS_VMAC if case["free"] == "eleven" else GUESS
            kw["numerics"], kw["stop_dchi2"] = case["numerics"], case["stop"]
            if case["start"] == "learned":
                kw["init_mode"], kw["mlp"] = G.INIT_LEARNED, _network(case["nl"])
        elif kind == "rois":
            kw["stop_dchi2"] = case["stop"]
        elif kind == "predict":
            net = _network(case["nl"])
        elif kind == "train":
            net = G.mlp_new(case["nl"], 3)
        eng.configure(G.make_config(LAMBDA0 + off, LAMBDA0, G.fe6173()[1], psf=taps, slight=stray, **kw))
        _kept[key] = (eng, off, taps, stray, net)
    return _kept[key]


def _regions(case):
    """Pixels and samples of each region of a batch: its layout, the same for every seed."""
    r = np.random.default_rng(case["layout"])
    return [(int(r.integers(case["side_min"], case["side_max"] + 1)) ** 2,
             int(r.integers(case["nl_min"], case["nl_max"] + 1))) for _ in range(case["rois"])]


def prepare(case, seed):
    eng, off, taps, stray, net = _engine(case)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    s = {"case": case, "eng": eng, "net": net}
    if case["kind"] == "rois":
        s["rois"] = []
        for n, nl in _regions(case):
            o = _grid(nl)
            t = _taps(o, case["psf"])
            s["rois"].append((_observe(_truth(n, g), o, t, None, g), LAMBDA0 + o, t))
        torch.cuda.synchronize()
        return s
    truth = _truth(case["pixels"], g, alpha=stray is not None)
    if case["kind"] == "synth":
        s["models"] = truth if case["f64"] else truth.float()
    else:
        obs = _observe(truth, off, taps, stray, g)
        s["obs"] = obs.cpu().numpy() if case.get("host") else obs
        if case["kind"] == "train":
            s["truth"] = truth
    torch.cuda.synchronize()
    return s


def run(state):
    case, eng = state["case"], state["eng"]
    kind = case["kind"]
    if kind == "synth":
        return eng.synthesize(state["models"], rf=case["rf"])
    if kind == "invert":
        return eng.invert(state["obs"])
    if kind == "rois":
        return eng.invert_rois(state["rois"])[0]
    if kind == "predict":
        return eng.mlp_predict(state["net"], state["obs"])
    net = G.Mlp()
    ctypes.pointer(net)[0] = state["net"]
    loss = eng.mlp_train(net, state["obs"], state["truth"], epochs=case["epochs"], batch=case["batch"])
    return {"loss": loss, **net.arrays()}


# ---------------------------------------------------------------- work and exact results
def work(case):
    """Bytes: inputs and outputs once.  Operations: the method's own count (profiles 385, response functions
    940, per sample and with the PSF 8 nl per row more), with the trials and accepted steps an inversion of such
    data takes (43 and 25; 16 and 10 with the early stop)."""
    def pixel(nl, psf, free, stop):
        trial = nl * 385 + (8 * nl * nl if psf else 0) + 24 * nl + free ** 3 / 3 + 2 * free ** 2
        acc = nl * 940 + (8 * nl * nl * (free - 1) if psf else 0) + 8 * nl * (free * (free + 3) / 2)
        t, a = (16, 10) if stop else (43, 25)
        return trial * (t + 1) + acc * (a + 1)

    kind = case["kind"]
    if kind == "rois":
        reg = _regions(case)
        return {"bytes": sum(n * (16 * nl + 56) for n, nl in reg),
                "flops": sum(n * pixel(nl, case["psf"], 9, case["stop"]) for n, nl in reg)}
    P, nl = case["pixels"], case["nl"]
    if kind == "synth":
        conv = 8 * nl * nl if case["psf"] else 0
        return {"bytes": P * ((88 if case["f64"] else 44) + 16 * nl * (11 if case["rf"] else 1)),
                "flops": P * (nl * 385 + conv + (nl * 870 + 8 * conv if case["rf"] else 0))}
    if kind == "invert":
        return {"bytes": P * (16 * nl + 132 + 16), "flops": P * pixel(nl, case["psf"], sum(FIX[case["free"]]), case["stop"])}
    mult = 4 * nl * 256 + 256 * 256 + 256 * 9
    if kind == "predict":
        return {"bytes": P * (16 * nl + 88), "flops": 2 * mult * P}
    n = case["epochs"] * (P // case["batch"]) * case["batch"]
    return {"bytes": n * (16 * nl + 88), "flops": 2 * n * (3 * mult - 4 * nl * 256)}


def exact(case, seed):
    if case["kind"] == "synth":
        eng, off, taps, stray, _ = _engine(case)
        m = prepare(case, seed)["models"].double()
        if not case["rf"]:
            return torch.cat([_profiles(c, off, taps, stray) for c in m.split(65536)])
        both = [_profiles(c, off, taps, stray, rf=True) for c in m.split(8192)]
        return tuple(torch.cat(x) for x in zip(*both))
    if case["kind"] == "predict":
        s = prepare(case, seed)
        a = {k: torch.tensor(v, dtype=torch.float64, device="cuda") for k, v in s["net"].arrays().items()}
        nl, x = case["nl"], torch.as_tensor(s["obs"]).cuda().double().reshape(case["pixels"], -1)
        h = (x - a["in_mean"][:4 * nl]) * a["in_scale"][:4 * nl]
        for w, b in ((a["w1"][:, :4 * nl], a["b1"]), (a["w2"], a["b2"])):
            h = torch.nn.functional.gelu(h @ w.T + b, approximate="tanh")
        y = (h @ a["w3"].T + a["b3"][:9]) * a["out_scale"][:9] + a["out_mean"][:9]
        lin = torch.hypot(y[:, 7], y[:, 8])
        az = 0.5 * torch.rad2deg(torch.atan2(y[:, 8], y[:, 7]))
        v = [y[:, 0].clamp(1, 2500), torch.hypot(y[:, 6], lin).clamp(max=5000), y[:, 1].clamp(-20, 20),
             y[:, 2].clamp(1e-4, 0.6), y[:, 3].clamp(1e-4, 10), torch.rad2deg(torch.atan2(lin, y[:, 6])),
             torch.where(az < 0, az + 180, az), y[:, 4].clamp(1e-4, 2), y[:, 5].clamp(1e-4, 2),
             torch.full_like(lin, GUESS[9]), torch.full_like(lin, GUESS[10])]
        out = torch.stack(v, dim=1)
        return out.cpu().numpy() if case["host"] else out
    return None
