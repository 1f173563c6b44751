"""Timing cases of the framework: what its users have it do, at the sizes they have it do it.

The workflow of an angle-domain Kirchhoff project runs through all of these: traveltime tables (``eikods``),
the migration of a survey into common-image gathers (``Plan.migrate``; ragged shots over depth windows as one
CUDA graph; leg fields from a learned surrogate), its adjoint (``Plan.model``), the datuming of the records
between depth windows (``datum_freq``) and the stitching of the windows' gathers (``stitch_windows``).

``listed()`` names one case of each, ``draw()`` gives others of the same ranges, ``prepare()`` makes what a
program has in hand before the call, ``run()`` is the call, ``work()`` what it cannot do without and
``exact()`` the same results in 64 bits from plain torch.  Lengths are in km, times in s.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import kirch_datuming_b200 as kd
from kirch_datuming_b200 import synth

F32, F64 = torch.float32, torch.float64
MUTE = ["direct_mute=1", "direct_mute_slope=0.5", "direct_mute_intercept=0", "direct_mute_taper=0.05"]
ANGLES = ["angle_min=0", "angle_max=60", "angle_step=1", "angle_n=61"]
#: the option sets that surveys are migrated with (tokens of the drop-in tools)
MODES = {
    "angle": ["cig=1", "mode=angle"] + ANGLES + MUTE,                                    # ADCIGs, two-bin
    "half": ["cig=1", "mode=angle", "half_angle=1", "angle_min=0", "angle_max=45", "angle_step=1.5", "angle_n=31"] + MUTE,
    "nearest": ["cig=1", "mode=angle", "angle_interp=0", "diff=1", "tau=0.01", "antialias=0.5", "aperture=60",
                "aperture_taper=5", "angle_taper_start=30", "angle_taper_end=50"] + ANGLES + MUTE,
    "offset": ["cig=1", "mode=offset"] + MUTE,                                           # offset-domain CIGs
    "stack": ["cig=0"] + MUTE,                                                           # the plain image
    "plain": ["aperture=60"],                                                            # kirchmig2d's stack
    "model": ["cig=1", "mode=angle", "adj=0"] + ANGLES,                                  # forward modelling
}


def listed():
    salt = dict(nz=601, nx=1601, d=0.01, npos=400, p0=0.0, dp=0.04)
    vz = dict(nz=201, nx=401, d=0.01, npos=401, p0=0.0, dp=0.01)
    return [
        # the smallest call: a test line on the fixtures' grid, where launches and host latency count
        dict(name="migrate_test_line", kind="migrate", mode="angle", interp="h", cmp=0, nz=41, nx=81, d=0.01, npos=41,
             p0=0.0, dp=0.02, ns=5, s0=0.05, ds=0.17, nh=21, h0=0.2, dh=0.02, nt=301, dt=0.002, surrogate=False),
        # a whole v(z) survey with a spread denser than its shots
        dict(vz, name="migrate_vz_survey", kind="migrate", mode="angle", interp="h", cmp=0, ns=64, s0=0.0, ds=4.0 / 63,
             nh=201, h0=1.0, dh=0.01, nt=1001, dt=0.002, surrogate=False),
        # the production size: a fixed spread that shoots from its own stations
        dict(salt, name="migrate_production", kind="migrate", mode="angle", interp="h", cmp=0, ns=400, s0=0.0, ds=0.04,
             nh=400, h0=0.0, dh=0.04, nt=3001, dt=0.001, surrogate=False),
        # a moving split spread: receivers belong to their shot, half-opening angles
        dict(vz, name="migrate_split_spread", kind="migrate", mode="half", interp="h", cmp=1, ns=48, s0=0.6, ds=0.06,
             nh=97, h0=-0.97, dh=0.02, nt=1001, dt=0.002, surrogate=False),
        # the same survey size with a learned traveltime surrogate in place of the tables
        dict(vz, name="migrate_surrogate", kind="migrate", mode="angle", interp="h", cmp=0, ns=64, s0=0.0, ds=4.0 / 63,
             nh=201, h0=1.0, dh=0.01, nt=1001, dt=0.002, surrogate=True),
        # uneven shots over the depth windows of the recursive workflow, replayed as one graph
        dict(name="windows_uneven", kind="windows", windows=3, rows=41, nx=401, d=0.01, shots=128, hmin=96, hmax=480,
             nrg=501, dh=0.008, tmin=1501, tmax=4001, dt=0.001),
        # forward modelling (adj=0) of a v(z) survey, the other half of a least-squares iteration
        dict(vz, name="model_vz", kind="model", mode="model", interp="h", cmp=0, ns=16, s0=0.1, ds=0.24, nh=101, h0=1.0,
             dh=0.02, nt=1001, dt=0.002, surrogate=False),
        # traveltime tables with source derivatives at every station of the production model
        dict(name="tables_production", kind="tables", nz=601, nx=1601, d=0.01, shots=400, order=2, derivs=True, grads=False),
        # tables of one depth window with the branch-aware gradients, first order
        dict(name="tables_window", kind="tables", nz=121, nx=401, d=0.01, shots=24, order=1, derivs=True, grads=True),
        # datuming of the production survey between two windows (fixed spread)
        dict(name="datum_production", kind="datum", cmp=0, ns=400, nh=400, nt=3001, dt=0.001, dx=0.04, datum=1.2,
             aperture=200, taper=0, data_taper=20, length=0.05),
        # datuming of a moving split spread (the tool's own default, cmp=1)
        dict(name="datum_split_spread", kind="datum", cmp=1, ns=64, nh=96, nt=751, dt=0.004, dx=0.02, datum=0.4,
             aperture=50, taper=10, data_taper=0, length=0.05),
        # stitching of five windows' gathers into the full-depth volume
        dict(name="stitch_production", kind="stitch", n1=601, n2=1601, n3=61, windows=5, overlap=20, blend=15, aper=50),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["migrate", "migrate", "migrate", "windows", "model", "tables", "datum", "datum", "stitch"])
    if kind in ("migrate", "model"):
        while True:
            small = kind == "model"
            nz, nx = _log(rng, 33, 301 if small else 601), _log(rng, 65, 601 if small else 1601)
            d, cmp = 0.01, rng.choice([0, 0, 1])
            ns, nh, dh = _log(rng, 4, 24 if small else 200), _log(rng, 8, 120 if small else 300), rng.choice([0.01, 0.02, 0.04])
            ext = (nx - 1) * d
            if cmp:
                h0, ds, s0 = -dh * (nh // 2), rng.choice([dh, 2 * dh]), 0.1 * ext
            elif rng.random() < 0.5:  # a spread that shoots from its own stations
                ds, h0 = dh, 0.0
                ns, s0 = min(ns, nh), dh * rng.randint(0, max(0, nh - min(ns, nh)))
            else:
                ds, h0, s0 = ext / max(1, ns - 1), rng.uniform(0.0, 0.3) * ext, 0.0
            # 5e9 pairs keep the 64-bit evaluation of a drawn case within seconds
            if ns * nh * nz * nx <= (3e8 if small else 5e9):
                break
        dp = rng.choice([0.02, 0.04])
        return dict(kind=kind, mode="model" if small else rng.choice(["angle", "angle", "half", "nearest", "offset", "stack", "plain"]),
                    interp=rng.choice(["h", "h", "l"]), cmp=cmp, nz=nz, nx=nx, d=d, npos=int(ext / dp) + 2, p0=0.0, dp=dp,
                    ns=ns, s0=s0, ds=ds, nh=nh, h0=h0, dh=dh, nt=_log(rng, 201, 2001), dt=rng.choice([0.002, 0.004]),
                    surrogate=not small and rng.random() < 0.1)
    if kind == "windows":
        return dict(kind=kind, windows=rng.randint(1, 3), rows=rng.randint(25, 61), nx=rng.randint(201, 601), d=0.01,
                    shots=_log(rng, 16, 128), hmin=rng.randint(24, 96), hmax=rng.randint(120, 400), nrg=501, dh=0.008,
                    tmin=rng.randint(501, 1501), tmax=rng.randint(1502, 4001), dt=0.001)
    if kind == "tables":
        return dict(kind=kind, nz=_log(rng, 41, 601), nx=_log(rng, 81, 1601), d=0.01, shots=_log(rng, 4, 300),
                    order=rng.choice([1, 2, 2]), derivs=rng.random() < 0.7, grads=rng.random() < 0.3)
    if kind == "datum":
        cmp = rng.choice([0, 0, 1])
        n = (lambda: _log(rng, 16, 96)) if cmp else (lambda: _log(rng, 24, 320))
        ns, nt = n(), _log(rng, 301, 1001 if cmp else 3001)
        dt = 0.004 if nt < 901 else rng.choice([0.002, 0.004])
        # a datum that the records reach well within their length
        return dict(kind=kind, cmp=cmp, ns=ns, nh=ns if not cmp and rng.random() < 0.5 else n(), nt=nt, dt=dt,
                    dx=rng.choice([0.02, 0.04]), datum=rng.uniform(0.2, min(1.2, 0.3 * nt * dt)), aperture=rng.randint(20, 60) if cmp else _log(rng, 20, 200),
                    taper=rng.choice([0, 3, 10]), data_taper=rng.choice([0, 5, 20]), length=rng.choice([0.025, 0.05, 0.1]))
    return dict(kind="stitch", n1=_log(rng, 101, 601), n2=_log(rng, 41, 1601), n3=rng.choice([1, 31, 61]),
                windows=rng.randint(2, 5), overlap=rng.randint(4, 20), blend=rng.choice([-1, 8, 15]), aper=rng.choice([0, 25, 50]))


# ---------------------------------------------------------------------------------------------- inputs --

def f32(v):
    """A header value as the tools read it: rounded to float."""
    return float(np.float32(v))


def _medium(seed):
    r = np.random.default_rng(seed)
    return float(r.uniform(1.4, 1.7)), float(r.uniform(0.45, 0.7))


def _arrival(v0, g, dx, z):
    """First arrival of v = v0 + g z from the surface over the lateral distance dx to depth z."""
    q = v0 * (v0 + g * z)
    e = g * g * (dx * dx + z * z) / (2.0 * q)
    return torch.log1p(e + torch.sqrt(e * (2.0 + e))) / g


def _tables(c, seed, z0=0.0):
    """Smooth traveltime tables [npos][nx][nz] and their derivative along the positions, FP32 on the device."""
    v0, g = _medium(seed)
    nz = c.get("nz", c.get("rows"))
    z = (z0 + torch.arange(nz, dtype=F64, device="cuda") * c["d"])[None, :]
    x = (torch.arange(c["nx"], dtype=F64, device="cuda") * c["d"])[:, None]
    ripple = 1.0 + 0.01 * torch.sin(3.0 * x + seed) * torch.sin(5.0 * z)
    T = torch.empty((c["npos"], c["nx"], nz), dtype=F32, device="cuda")
    D = torch.empty_like(T)
    for k in range(c["npos"]):
        dx = x - (c["p0"] + k * c["dp"])
        q = v0 * (v0 + g * z)
        r = torch.sqrt(dx * dx + z * z)
        e = g * g * r * r / (2.0 * q)
        T[k] = (_arrival(v0, g, dx, z) * ripple).float()
        slope = -dx / torch.clamp(r, min=1e-9) * torch.sqrt(2.0 / (q * (2.0 + e)))
        D[k] = (slope * ripple).float()
    return T, D


def _gathers(offsets, nt, dt, seed, freq):
    """Seeded records: reflection hyperbolas with a Ricker wavelet and noise 20 dB below, [offsets..., nt]."""
    r = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.arange(nt, dtype=F32, device="cuda") * dt
    out = torch.empty((*offsets.shape, nt), dtype=F32, device="cuda")
    ev = [(r.uniform(0.15, 0.8) * nt * dt, r.uniform(1.6, 3.0), r.uniform(0.05, 0.2) * (1 if r.random() < 0.5 else -1))
          for _ in range(4)]
    for i in range(offsets.shape[0]):
        acc = torch.randn(out[i].shape, generator=gen, dtype=F32, device="cuda") * 0.01
        for t0, v, a in ev:
            tt = torch.sqrt(t0 * t0 + (offsets[i] / v) ** 2)[..., None]
            acc += a * synth.ricker(t - tt, freq)
        out[i] = acc
    return out


def _geometry(c):
    g = dict(nt=c["nt"], nh=c["nh"], ns=c["ns"], t0=0.0, dt=f32(c["dt"]), h0=f32(c["h0"]), dh=f32(c["dh"]), s0=f32(c["s0"]),
             ds=f32(c["ds"]), nz=c["nz"], nx=c["nx"], z0=0.0, dz=f32(c["d"]), x0=0.0, dx=f32(c["d"]))
    for s in "sr":
        g.update({s + "ny": c["npos"], s + "y0": f32(c["p0"]), "%sdy" % s: f32(c["dp"])})
    return g


def _axis(c):
    """(bins, first, step) of the output axis of a case's mode."""
    if c["mode"] == "offset":
        return c["nh"], min(f32(c["h0"]), f32(c["h0"] + (c["nh"] - 1) * c["dh"])), abs(f32(c["dh"]))
    return {"half": (31, 0.0, 1.5), "stack": (1, 0.0, 1.0), "plain": (1, 0.0, 1.0)}.get(c["mode"], (61, 0.0, 1.0))


def _params(c):
    if c["mode"] == "plain":
        return kd.params_kirchmig2d(*MODES["plain"], "cmp=%d" % c["cmp"], "type=%s" % c["interp"])
    return kd.params(*MODES[c["mode"]], "cmp=%d" % c["cmp"], "type=%s" % c["interp"])


def _offsets(c):
    s = c["s0"] + torch.arange(c["ns"], dtype=F32, device="cuda") * c["ds"]
    h = c["h0"] + torch.arange(c["nh"], dtype=F32, device="cuda") * c["dh"]
    return h[None, :].abs().expand(c["ns"], -1) if c["cmp"] else (h[None, :] - s[:, None]).abs()


def _model_image(c, ng, seed):
    """Layered reflectivity with lateral and angle variation, [ng][nx][nz]."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    base = torch.randn((1, 1, c["nz"]), generator=gen, dtype=F32, device="cuda")
    return (base * 0.1 + 0.02 * torch.randn((ng, c["nx"], c["nz"]), generator=gen, dtype=F32, device="cuda")).contiguous()


def _surrogate(c, seed):
    """A network over the survey's domain, and its parameters (FP32)."""
    v0, g = _medium(seed)
    ext, dep = (c["nx"] - 1) * c["d"], (c["nz"] - 1) * c["d"]
    net = kd.Surrogate((0.0, 0.0, 0.0), (ext, dep, ext), fmax=3.0, vref=v0, zsrc=0.0, seed=seed, vgrad=g, residual_ms=1.0)
    return net


def _uneven(c, seed):
    """The uneven shots of one survey: positions, first stations, receiver counts and trace lengths."""
    r = np.random.default_rng(seed)
    n = c["shots"]
    nh, nt = r.integers(c["hmin"], c["hmax"] + 1, n), r.integers(c["tmin"], c["tmax"] + 1, n)
    ext = (c["nx"] - 1) * c["d"]
    sx = (np.arange(n) * (ext / max(1, n - 1))).astype(np.float32)
    i0 = np.clip(np.round((sx - nh * c["dh"] / 2) / c["dh"]).astype(int), 0, c["nrg"] - nh)
    return sx, i0, nh, nt


def _window(c, w):
    """Case of depth window w: its own tables start at the window's top."""
    return dict(c, nz=c["rows"], npos=c["nx"], p0=0.0, dp=c["d"])


def _window_shots(c, seed, w):
    sx, i0, nh, nt = _uneven(c, seed)
    grid = (np.arange(c["nrg"]) * c["dh"]).astype(np.float32)
    shots = []
    for s in range(c["shots"]):
        h = grid[i0[s]:i0[s] + nh[s]]
        off = torch.from_numpy(np.abs(h - sx[s])).cuda()
        shots.append(dict(sx=float(sx[s]), dh=c["dh"], h=h,
                          data=_gathers(off[None], int(nt[s]), c["dt"], seed * 1000 + 131 * w + s, 20.0)[0]))
    return shots


def _rows(c):
    """(start, end) of the stitched windows."""
    n, ov = c["windows"], c["overlap"]
    cut = [round(k * (c["n1"] - 1) / n) for k in range(n + 1)]
    return [(max(0, cut[k] - (ov if k else 0)), cut[k + 1]) for k in range(n)]


def _stitch_scales(c):
    return [f32(1.0 + 0.1 * (k % 3) - 0.05 * k) for k in range(c["windows"])]


def _datum_case(c, seed):
    """(parameters, table, records) of a datuming call: one table serves both sides, as the workflow has it."""
    dx, ns, nh = c["dx"], c["ns"], c["nh"]
    if c["cmp"]:
        half = nh // 2
        ng, g0 = ns + nh + 2, 0.0
        s0, h0 = dx * (half + 1), -dx * half
    else:
        ng, g0, s0, h0 = max(ns, nh), 0.0, 0.0, 0.0
    p = dict(nt=c["nt"], nh=nh, ns=ns, dt=f32(c["dt"]), h0=f32(h0), dh=f32(dx), s0=f32(s0), ds=f32(dx), nsg=ng, nrg=ng,
             sg0=f32(g0), dsg=f32(dx), rg0=f32(g0), drg=f32(dx), sdatum=f32(c["datum"]), rdatum=f32(c["datum"]),
             aperture=c["aperture"], taper=c["taper"], data_taper=c["data_taper"], length=f32(c["length"]), antialias=1.0,
             cmp=c["cmp"])
    v0, g = _medium(seed)
    x = torch.arange(ng, dtype=F64, device="cuda") * dx
    z = torch.full((1, 1), c["datum"], dtype=F64, device="cuda")
    table = _arrival(v0, g, x[:, None] - x[None, :], z).float().contiguous()
    s = s0 + torch.arange(ns, dtype=F32, device="cuda") * dx
    h = h0 + torch.arange(nh, dtype=F32, device="cuda") * dx
    off = h[None, :].abs().expand(ns, -1) if c["cmp"] else (h[None, :] - s[:, None]).abs()
    return p, table, _gathers(off, c["nt"], c["dt"], seed, 15.0)


# ------------------------------------------------------------------------------------------ the calls --

def prepare(case, seed):
    c = case
    if c["kind"] in ("migrate", "model"):
        plan = kd.Plan(_params(c), kd.geometry(**_geometry(c)), 40 << 30)
        T, D = _tables(c, seed)
        plan.set_tables(T, D)
        if c["surrogate"]:
            net = _surrogate(c, seed)
            plan.set_surrogate(net, net)
        if c["kind"] == "model":
            out = torch.zeros((c["ns"], c["nh"], c["nt"]), dtype=F32, device="cuda")
            return dict(kind="model", plan=plan, image=_model_image(c, plan.ng, seed), out=out)
        out = torch.zeros((plan.ng, c["nx"], c["nz"]), dtype=F32, device="cuda")
        return dict(kind="migrate", plan=plan, data=_gathers(_offsets(c), c["nt"], c["dt"], seed, 15.0), out=out)
    if c["kind"] == "windows":
        plans, images = [], []
        for w in range(c["windows"]):
            cw = _window(c, w)
            g = _geometry(dict(cw, nt=c["tmax"], nh=1, ns=1, h0=0.0, s0=0.0, ds=0.0))
            plan = kd.Plan(kd.params(*MODES["angle"], "cmp=0"), kd.geometry(**g), 12 << 30)
            T, D = _tables(cw, seed + w)
            plan.set_tables(T, D)
            plan.prepare_shots(_window_shots(c, seed, w))
            plans.append(plan)
            images.append(torch.zeros((plan.ng, c["nx"], c["rows"]), dtype=F32, device="cuda"))
        torch.cuda.synchronize()
        return dict(kind="windows", graph=kd.Graph(plans, images), images=images)
    if c["kind"] == "tables":
        v, _ = synth.five_layer_salt(c["nz"], c["nx"], c["d"], c["d"], seed=seed)
        x = np.linspace(0.0, (c["nx"] - 1) * c["d"], c["shots"] + 2)[1:-1] if c["shots"] < c["nx"] else None
        x = np.arange(c["shots"]) * c["d"] * (c["nx"] - 1) / max(1, c["shots"]) if x is None else x
        shots = np.zeros((c["shots"], 3), np.float32)
        shots[:, 1] = x
        return dict(kind="tables", vel=torch.from_numpy(v).cuda(), shots=shots, c=c)
    if c["kind"] == "datum":
        p, table, data = _datum_case(c, seed)
        return dict(kind="datum", p=kd.datum_params(**p), table=table, data=data, out=torch.empty_like(data))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    layers = [torch.randn((c["n3"], c["n2"], e - s + 1), generator=gen, dtype=F32, device="cuda") for s, e in _rows(c)]
    return dict(kind="stitch", c=c, layers=layers, out=torch.empty((c["n3"], c["n2"], c["n1"]), dtype=F32, device="cuda"))


def run(state):
    s = state
    if s["kind"] == "migrate":
        return s["plan"].migrate(s["data"], s["out"])
    if s["kind"] == "model":
        return s["plan"].model(s["image"], s["out"])
    if s["kind"] == "windows":
        s["graph"].launch()
        return s["images"]
    if s["kind"] == "tables":
        c = s["c"]
        return kd.eikods(s["vel"], c["d"], c["d"], s["shots"], order=c["order"], derivs=c["derivs"], grads=c["grads"])
    if s["kind"] == "datum":
        return kd.datum_freq(s["p"], s["table"], s["table"], s["data"], s["out"])
    c = s["c"]
    bad = kd.stitch_windows(s["out"], s["layers"], _rows(c), c["blend"], _stitch_scales(c), True, c["aper"], 1.5)
    return [s["out"], bad]


def work(case):
    c = case
    if c["kind"] in ("migrate", "model"):
        pairs = c["ns"] * c["nh"] * c["nz"] * c["nx"]
        ng = _axis(c)[0]
        b = 4 * (2 * c["npos"] * c["nx"] * c["nz"] + c["ns"] * c["nh"] * c["nt"] + ng * c["nx"] * c["nz"])
        # a pair: the two legs' times and directions combined (4), the bin and its weights (6), three picks of the
        # trace (sample position, fraction, interpolation: 12), the pick's weight (5), one or two bins updated (4)
        f = 31.0 * pairs
        if c["surrogate"]:  # 384-128-128-128-128-1 forward, and back to the source position, at every leg point
            f += (c["ns"] + c["nh"]) * c["nz"] * c["nx"] * 2.0 * (256 * 128 + 3 * 128 * 128 + 3 * 128 * 128)
        return dict(bytes=b, flops=f)
    if c["kind"] == "windows":
        h, t = (c["hmin"] + c["hmax"]) / 2, (c["tmin"] + c["tmax"]) / 2
        n = c["rows"] * c["nx"]
        return dict(bytes=4.0 * c["windows"] * (2 * c["nx"] * n + c["shots"] * h * t + 61 * n),
                    flops=31.0 * c["windows"] * c["shots"] * h * n)
    if c["kind"] == "tables":
        n = c["shots"] * c["nz"] * c["nx"]
        outs = 1 + 2 * c["derivs"] + 2 * c["grads"]
        return dict(bytes=4.0 * (n * outs + c["nz"] * c["nx"]), flops=n * (40.0 + 40.0 * c["derivs"]))
    if c["kind"] == "datum":
        near = lambda n: sum(min(n - 1, i + c["aperture"]) - max(0, i - c["aperture"]) + 1 for i in range(n))  # noqa: E731
        nf = c["nt"]  # at least as many frequencies as half the samples of a doubled trace
        terms = near(c["nh"]) * c["ns"] + near(c["ns"]) * c["nh"]
        return dict(bytes=8.0 * c["ns"] * c["nh"] * c["nt"], flops=8.0 * terms * nf)
    win = sum(e - s + 1 for s, e in _rows(c))
    return dict(bytes=4.0 * c["n2"] * c["n3"] * (win + c["n1"]), flops=2.0 * c["n2"] * c["n3"] * win)


# ------------------------------------------------------------------------------ the same in 64 bits --

class _Leg64:
    """Leg fields in 64 bits; the slice a position falls in is decided in float, as the tools decide it."""

    def __init__(self, c, seed, T, D, plain):
        self.c, self.T, self.D, self.plain = c, T, D, plain
        self.g = _geometry(c)
        self.ap = {"nearest": (60.0, 5.0), "plain": (60.0, 0.0)}.get(c["mode"], (90.0, 10.0))
        self.net = _Net64(c, seed) if c.get("surrogate") else None
        dz, dx = self.g["dz"], self.g["dx"]
        self.z = torch.arange(c["nz"], dtype=F64, device="cuda")[None, :] * dz
        self.x = torch.arange(c["nx"], dtype=F64, device="cuda")[:, None] * dx

    def table(self, pos, posf):
        c, g = self.c, self.g
        n, o, d = c["npos"], np.float32(g["sy0"]), np.float32(g["sdy"])
        f = (np.float32(posf) - o) / d
        i0 = int(f) if self.plain else int(math.floor(f))
        if (i0 <= 0 if self.plain else f <= 0):
            return self.T[0].double(), self.D[0].double()
        if f >= n - 1 or i0 >= n - 1:
            return self.T[n - 1].double(), self.D[n - 1].double()
        d = float(d)
        t = (pos - (float(o) + i0 * d)) / d
        p0, p1, m0, m1 = self.T[i0].double(), self.T[i0 + 1].double(), self.D[i0].double(), self.D[i0 + 1].double()
        if c["interp"] == "l":
            return (1 - t) * p0 + t * p1, (p1 - p0) / d
        return ((2 * t ** 3 - 3 * t * t + 1) * p0 + (t ** 3 - 2 * t * t + t) * d * m0 + (3 * t * t - 2 * t ** 3) * p1
                + (t ** 3 - t * t) * d * m1,
                -6 * t * (1 - t) / d * (p0 - p1) + (1 - t) * (1 - 3 * t) * m0 + (3 * t * t - 2 * t) * m1)

    @staticmethod
    def _diff(a, dim, step):
        n = a.shape[dim]
        i = torch.arange(n, device="cuda")
        lo, hi = (i - 2).clamp(min=0), (i + 2).clamp(max=n - 1)
        span = ((hi - lo).double() * step).view(-1, 1) if dim == 0 else ((hi - lo).double() * step).view(1, -1)
        return (a.index_select(dim, hi) - a.index_select(dim, lo)) / span

    @staticmethod
    def _box(a, dim):
        n = a.shape[dim]
        i = torch.arange(n, device="cuda")
        s, k = torch.zeros_like(a), torch.zeros(n, dtype=F64, device="cuda")
        for o in range(-2, 3):
            ok = ((i + o >= 0) & (i + o < n)).double()
            s += a.index_select(dim, (i + o).clamp(0, n - 1)) * (ok.view(-1, 1) if dim == 0 else ok.view(1, -1))
            k += ok
        return s / (k.view(-1, 1) if dim == 0 else k.view(1, -1))

    def __call__(self, pos, posf, scale):
        """(T, phi, Tx * scale, aperture weight) over the grid, flat."""
        T, Tx = self.net(pos, self.z, self.x) if self.net else self.table(pos, posf)
        if self.plain:
            left = torch.rad2deg(torch.atan((pos - self.x) / self.z)) > self.ap[0]
            right = torch.rad2deg(torch.atan((self.x - pos) / self.z)) > self.ap[0]
            w = (~left).double() + 2.0 * (~right).double()
        else:
            deg = torch.rad2deg(torch.atan((pos - self.x).abs() / self.z.abs().clamp(min=1e-12)))
            a, b = self.ap
            u = ((deg - (a - b)) / b).clamp(0, 1)
            w = 0.5 * (1 + torch.cos(math.pi * u))
        phi = None
        if self.c["mode"] in ("angle", "half", "nearest", "model"):
            gx, gz = self._diff(T, 0, self.g["dx"]), self._diff(T, 1, self.g["dz"])
            for _ in range(2):
                gx, gz = (self._box(self._box(v, 1), 0) for v in (gx, gz))
            phi = torch.where(torch.sqrt(gx * gx + gz * gz) <= 1e-12, math.nan, torch.atan2(gz, gx)).reshape(-1)
        return T.reshape(-1), phi, (Tx * scale).reshape(-1), w.reshape(-1)


class _Net64:
    """The surrogate's traveltime and its source derivative: the network on 3 x 64 Fourier features, in 64 bits."""

    def __init__(self, c, seed):
        net = _surrogate(c, seed)
        p = torch.from_numpy(net.get_params()).cuda().double()
        net.close()
        self.v0, self.g = _medium(seed)
        self.v0, self.g = f32(self.v0), f32(self.g)
        H, F = 128, 384
        n = [H * F, H * H, H * H, H * H, H, H, H, H, H, 1]
        parts = torch.split(p, n)
        self.W = [parts[0].view(H, F)] + [w.view(H, H) for w in parts[1:4]]
        self.b, self.wo, self.bo = parts[4:8], parts[8], parts[9]
        ext, dep = f32((c["nx"] - 1) * c["d"]), f32((c["nz"] - 1) * c["d"])
        self.scale = [2.0 / v for v in (ext, dep, ext)]
        self.k = torch.arange(1, 65, dtype=F64, device="cuda") * (math.pi * 3.0 / 64)

    def __call__(self, pos, z, x):
        shape = (x.shape[0], z.shape[1])
        Z, X = z.expand(shape).reshape(-1), x.expand(shape).reshape(-1)
        T, Tx = torch.empty_like(Z), torch.empty_like(Z)
        for a in range(0, Z.numel(), 1 << 16):
            T[a:a + (1 << 16)], Tx[a:a + (1 << 16)] = self._eval(pos, Z[a:a + (1 << 16)], X[a:a + (1 << 16)])
        return T.view(shape), Tx.view(shape)

    def _eval(self, pos, z, x):
        feats, dxs = [], None
        for i, v in enumerate((torch.full_like(z, pos), z, x)):
            th = (v * self.scale[i] - 1.0)[:, None] * self.k
            feats.append(torch.stack([torch.sin(th), torch.cos(th)], -1).flatten(1))
            if i == 0:
                dxs = torch.stack([self.k * torch.cos(th), -self.k * torch.sin(th)], -1).flatten(1)
        h, hd = torch.cat(feats, 1) @ self.W[0].T + self.b[0], dxs @ self.W[0][:, :128].T
        for layer in range(4):
            s = torch.sigmoid(h)
            h, hd = h * s, hd * s * (1.0 + h * (1.0 - s))
            if layer < 3:
                h, hd = h @ self.W[layer + 1].T + self.b[layer + 1], hd @ self.W[layer + 1].T
        out, dout = h @ self.wo + self.bo, (hd @ self.wo) * self.scale[0]
        dxv, q = x - pos, self.v0 * (self.v0 + self.g * z)
        r = torch.sqrt(dxv * dxv + z * z)
        e = self.g * self.g * r * r / (2.0 * q)
        k = torch.where(r > 0, torch.sqrt(2.0 / (q * (2.0 + e))) / torch.clamp(r, min=1e-300), 0.0)
        return _arrival(self.v0, self.g, dxv, z) + 1e-3 * out, -dxv * k + 1e-3 * dout


class _Pairs64:
    """The gates, bins and picks of one shot against its receivers in 64 bits (arrays [nh][points])."""

    def __init__(self, c, ng, g0, dg):
        self.c, self.ng, self.g0, self.dg = c, ng, float(g0), float(dg)
        self.tau, self.aal = (f32(0.01), 0.5) if c["mode"] == "nearest" else (0.0, 1.0)
        zf = torch.arange(c["nz"], dtype=F64, device="cuda") / max(1, c["nz"] - 1)
        lo, hi = (40.0, 25.0) if c["mode"] == "half" else (80.0, 50.0)
        self.cut = (lo + zf * (hi - lo)).expand(c["nx"], -1).reshape(-1)[None, :]

    def __call__(self, s, r, nt, bins=None, src_left=None):
        """s: the shot's leg; r: stacked receiver legs -> (keep, bin, weight of bin, weight of bin + 1, positions,
        pick weight); bins: the offset bins, src_left: kirchmig2d's side of each trace."""
        m, dt = self.c["mode"], f32(self.c["dt"])
        if m == "plain":
            sl, rl = s[3][None, :], r[3]
            both = lambda left, right: ((left % 2) >= 1) & (right >= 2)  # noqa: E731
            keep = torch.where(src_left[:, None], both(sl, rl), both(rl, sl))
            w = torch.ones_like(r[0])
        else:
            w = s[3][None, :] * r[3]
            keep = w > 0
        b, w1 = (bins[:, None].expand_as(w) if bins is not None else torch.zeros_like(w, dtype=torch.long)), torch.zeros_like(w)
        if m in ("angle", "half", "nearest", "model"):
            th = (s[1][None, :] - r[1]).abs()
            th = torch.where(th > math.pi, 2 * math.pi - th, th)
            ang = th * ((90.0 if m == "half" else 180.0) / math.pi)
            u = (ang - self.g0) / self.dg
            top = self.ng - 1
            if m == "nearest":
                fl = torch.floor(u + 0.5)
                keep &= (fl >= 0) & (fl <= top)
                b = torch.nan_to_num(fl).long().clamp(0, top)
                w = w * 0.5 * (1 + torch.cos(math.pi * ((ang - 30.0) / 20.0).clamp(0, 1)))
            else:
                keep &= (u >= -1e-5) & (u <= top + 1e-5)
                uc = torch.nan_to_num(u).clamp(0, top)
                b = uc.floor().long()
                w1 = uc - b
            w = w * 0.5 * (1 + torch.cos(math.pi * ((ang - self.cut) / 10.0).clamp(0, 1)))
            keep &= w > 0
        f0 = (s[0][None, :] + r[0] + self.tau) / dt
        half = 1.0 + torch.maximum(s[2].abs()[None, :], r[2].abs()) * (self.aal / dt)
        keep &= (f0 - half >= 0) & (f0 + half < nt - 1)
        return keep, b, 1.0 - w1, w1, (f0, f0 - half, f0 + half), w / (1.0 + 2.0 * half) ** 2


def _doubint(x):
    return torch.flip(torch.cumsum(torch.flip(torch.cumsum(x, -1), [-1]), -1), [-1])


def _traces64(c, data, off, mute):
    """Integrated traces of one shot in 64 bits; off: the offsets of its receivers."""
    x, dt = data.double(), f32(c["dt"])
    if mute:
        t = torch.arange(x.shape[-1], dtype=F64, device="cuda")[None, :] * dt
        u = ((t - 0.5 * off[:, None]) / f32(0.05)).clamp(0, 1)
        x = x * (0.5 * (1 - torch.cos(math.pi * u)))
    x = _doubint(x)
    if c["mode"] == "nearest":
        y = torch.empty_like(x)
        y[:, 1:-1] = (x[:, 2:] - x[:, :-2]) / (2 * dt)
        y[:, 0], y[:, -1] = (x[:, 1] - x[:, 0]) / dt, (x[:, -1] - x[:, -2]) / dt
        x = y
    return x


def _pick64(D, pos, keep):
    """2 D(f0) - D(f-) - D(f+), linear between samples."""
    out = 0.0
    for f, k in zip(pos, (2.0, -1.0, -1.0)):
        f = torch.where(keep, f, 0.0)
        i = f.floor().long()
        a = torch.gather(D, 1, i)
        out = out + k * (a + (f - i) * (torch.gather(D, 1, i + 1) - a))
    return out


def _survey64(c, seed, shots, ng, g0, dg, T, D, sink):
    """Every shot's pairs to sink(k, offsets, pairs): shots is a list of (position, float position, receiver
    positions, float receiver positions, ds, dh, nt, bins, source-left flags)."""
    leg = _Leg64(c, seed, T, D, c["mode"] == "plain")
    pairs = _Pairs64(c, ng, g0, dg)
    kept = {}

    def receiver(p, pf, dh):
        if (p, float(pf), dh) not in kept:
            if len(kept) > 600:
                kept.clear()
            kept[(p, float(pf), dh)] = leg(p, pf, dh)
        return kept[(p, float(pf), dh)]

    for k, (sx, sxf, rx, rxf, ds, dh, nt, bins, left) in enumerate(shots):
        s = leg(sx, sxf, ds)
        step = max(1, int(4e7) // (c["nz"] * c["nx"]))
        for a in range(0, len(rx), step):
            b = min(len(rx), a + step)
            legs = [receiver(rx[j], rxf[j], dh) for j in range(a, b)]
            r = [None if legs[0][q] is None else torch.stack([v[q] for v in legs]) for q in range(4)]
            sel = lambda v: None if v is None else v[a:b]  # noqa: E731
            off = torch.tensor([abs(v - sx) for v in rx[a:b]], dtype=F64, device="cuda")
            sink(k, a, b, off, pairs(s, r, nt, sel(bins), sel(left)))


def _survey_shots(c, ng, g0, dg):
    g = _geometry(c)
    out = []
    for k in range(c["ns"]):
        ds, dh = (g["ds"] if c["ns"] > 1 else 0.0), (g["dh"] if c["nh"] > 1 else 0.0)
        sx, sxf = g["s0"] + k * ds, np.float32(g["s0"]) + np.float32(k) * np.float32(ds)
        h = [g["h0"] + j * dh for j in range(c["nh"])]
        hf = np.float32(g["h0"]) + np.arange(c["nh"], dtype=np.float32) * np.float32(dh)
        rx, rxf = ([sx + v for v in h], sxf + hf) if c["cmp"] else (h, hf)
        bins = left = None
        if c["mode"] == "offset":
            bins = torch.from_numpy(np.floor((hf - np.float32(g0)) / np.float32(dg) + np.float32(0.5)).astype(np.int64)).cuda()
        if c["mode"] == "plain":
            left = torch.from_numpy(hf >= 0 if c["cmp"] else hf - sxf >= 0).cuda()
        out.append((sx, sxf, rx, rxf, ds, dh, c["nt"], bins, left))
    return out


def _image64(c, seed, shots, ng, g0, dg, T, D, data):
    """The image of shots whose records are data[k], in 64 bits."""
    n = c["nz"] * c["nx"]
    img = torch.zeros(ng * n, dtype=F64, device="cuda")
    pt = torch.arange(n, device="cuda")[None, :]

    def sink(k, a, b, off, found):
        keep, bin_, w0, w1, pos, aw = found
        tr = _traces64(c, data[k][a:b], off, c["mode"] != "plain")
        v = torch.where(keep, _pick64(tr, pos, keep) * aw, 0.0)
        img.index_add_(0, (bin_ * n + pt).reshape(-1), (v * w0).reshape(-1))
        up = (keep & (w1 > 0)).double()
        img.index_add_(0, ((bin_ + (w1 > 0)).clamp(max=ng - 1) * n + pt).reshape(-1), (v * w1 * up).reshape(-1))

    _survey64(c, seed, shots, ng, g0, dg, T, D, sink)
    return img.view(ng, c["nx"], c["nz"])


def _model64(c, seed):
    """Forward modelling in 64 bits: the picks run backwards."""
    ng, g0, dg = _axis(c)
    T, D = _tables(c, seed)
    image = _model_image(c, ng, seed).double().view(ng, -1)
    out = torch.zeros((c["ns"], c["nh"], c["nt"]), dtype=F64, device="cuda")

    def sink(k, a, b, off, found):
        keep, bin_, w0, w1, pos, aw = found
        m = w0 * torch.gather(image, 0, bin_) + w1 * torch.gather(image, 0, (bin_ + 1).clamp(max=ng - 1))
        v = torch.where(keep, m * aw, 0.0)
        raw = torch.zeros(((b - a) * c["nt"]), dtype=F64, device="cuda")
        row = torch.arange(b - a, device="cuda")[:, None] * c["nt"]
        for f, s in zip(pos, (2.0, -1.0, -1.0)):
            f = torch.where(keep, f, 0.0)
            i = f.floor().long()
            raw.index_add_(0, (row + i).reshape(-1), (s * v * (1 - (f - i))).reshape(-1))
            raw.index_add_(0, (row + i + 1).reshape(-1), (s * v * (f - i)).reshape(-1))
        out[k, a:b] = _doubint(raw.view(b - a, c["nt"]))

    _survey64(c, seed, _survey_shots(c, ng, g0, dg), ng, g0, dg, T, D, sink)
    return out


def _filter64(tau, slope, w, p, nfft, iw):
    """Operator terms w aa(iw) H(tau, iw) in 64 bits, [iw][...]: the half-derivative filter's samples are second
    differences of sqrt(t^2 - 1), placed at tau between two samples."""
    dt = p["dt"]
    K = int(np.float32(p["length"]) / np.float32(dt)) + 1
    tau = tau.double()
    ts = torch.where(tau > 0, tau, 1.0)
    u = torch.arange(1, K + 1, dtype=F64, device="cuda") * (dt / ts[..., None])
    r = torch.sqrt(u * (2 + u))
    r = torch.nn.functional.pad(r, (2, 0))
    F = (r[..., 2:] - 2 * r[..., 1:-1] + r[..., :-2]) / dt
    k = torch.arange(K, device="cuda")
    unit = lambda n: torch.polar(torch.ones((), dtype=F64, device="cuda"), -2 * math.pi / nfft * (n % nfft).double())  # noqa: E731
    E = unit(iw[:, None] * k[None, :])
    Ff = F.reshape(-1, K)
    S = torch.complex(E.real @ Ff.T, E.imag @ Ff.T).view(iw.numel(), *tau.shape)
    m = torch.ceil(ts / dt)
    d = m - ts / dt
    ph = iw.view(-1, *[1] * tau.dim()) * m.long()
    lin = unit(ph) * ((1 - d) + d * unit(-iw).view(-1, *[1] * tau.dim()))
    fmax = 0.5 / (slope.double().abs() * p["antialias"])
    freq = (iw.double() / (nfft * dt)).view(-1, *[1] * tau.dim())
    x = ((freq - 0.8 * fmax) / (0.2 * fmax)).clamp(0, 1)
    act = (slope.abs() > 1e-12) & (fmax < 0.5 / dt)
    aa = torch.where(act & (freq > 0), 0.5 * (1 + torch.cos(math.pi * x)), 1.0)
    return S * lin * (aa * torch.where(tau > 0, w, 0.0))


def _edge(n, tap):
    i = np.arange(n)
    t = min(tap, (n - 1) // 2)
    if t <= 0:
        return np.ones(n)
    return 0.5 * (1 - np.cos(np.pi * np.minimum(1.0, np.minimum(i, n - 1 - i) / t)))


def _side(n, step, datum, aper, tap, scale=1.0):
    """Weights [out][in] of one side without tau: taper times step datum / (pi distance^2)."""
    i, j = np.arange(n)[:, None], np.arange(n)[None, :]
    left, right = np.maximum(0, i - aper), np.minimum(n - 1, i + aper)
    inside = (j >= left) & (j <= right)
    w = np.where(inside, 1.0, 0.0)
    if tap > 0:
        for e in ((j - left) / tap, (right - j) / tap):
            w = w * 0.5 * (1 - np.cos(np.pi * np.clip(e, 0, 1)))
    return torch.from_numpy(w * step * datum / math.pi / (datum * datum + (j - i) ** 2 * step * step)).cuda()


def _slope(table, d):
    t = table.double()
    s = torch.empty_like(t)
    s[1:-1] = 0.5 * (t[2:] - t[:-2]) / d
    s[0], s[-1] = (t[1] - t[0]) / d, (t[-1] - t[-2]) / d
    return s


def _datum64(c, seed):
    """Datuming in 64 bits: per frequency, the receiver side and then the source side as dense sums."""
    p, table, data = _datum_case(c, seed)
    ns, nh, nt, dx = p["ns"], p["nh"], p["nt"], p["dh"]
    steps = math.ceil(float(np.float32(table.max().item()) / np.float32(p["dt"])))
    need, nfft = nt + steps + int(np.float32(p["length"]) / np.float32(p["dt"])) + 2, 1
    while nfft < need:
        nfft *= 2
    nw = nfft // 2 + 1
    wt = torch.from_numpy(np.outer(_edge(ns, p["data_taper"]), _edge(nh, p["data_taper"]))).cuda()
    U = torch.empty((nw, ns, nh), dtype=torch.complex128, device="cuda")
    for s in range(0, ns, 8):
        x = torch.flip(data[s:s + 8].double(), [-1]) * wt[s:s + 8, :, None]
        U[:, s:s + 8] = torch.fft.rfft(x, n=nfft).permute(2, 0, 1)
    ap, tap, ng, dat = c["aperture"], c["taper"], p["nrg"], p["rdatum"]
    sl = _slope(table, dx) * dx
    Wr, Ws = _side(nh, dx, dat, ap, tap), _side(ns, dx, dat, ap, tap)
    cr = np.array([[int(((s if c["cmp"] else np.float32(0)) + np.float32(p["h0"]) + np.float32(j) * np.float32(dx)
                         - np.float32(p["rg0"])) / np.float32(dx) + np.float32(0.5)) for j in range(nh)]
                   for s in (np.float32(p["s0"]) + np.arange(ns if c["cmp"] else 1, dtype=np.float32) * np.float32(dx))])
    cs = np.array([int((np.float32(p["s0"]) + np.float32(i) * np.float32(dx) - np.float32(p["sg0"])) / np.float32(dx)
                       + np.float32(0.5)) for i in range(ns)])
    ti = lambda a: torch.from_numpy(np.asarray(a)).cuda()  # noqa: E731
    step = max(1, min(256, int(4e9) // (16 * max(ng * ng, ns * nh))))
    for f in range(0, nw, step):
        iw = torch.arange(f, min(nw, f + step), device="cuda")
        if not c["cmp"]:
            at = lambda i: (table[i[None, :], i[:, None]], sl[i[None, :], i[:, None]])  # noqa: E731
            (tr, sr), (ts, ss) = at(ti(cr[0])), at(ti(cs))
            Kr, Ks = _filter64(tr, sr, Wr * tr.double(), p, nfft, iw), _filter64(ts, ss, Ws * ts.double(), p, nfft, iw)
            U[f:f + step] = Ks @ (U[f:f + step] @ Kr.transpose(1, 2))
            continue
        # cmp=1: the operators of every table pair, then the sums of each shot and of each common-receiver gather
        H = _filter64(table, sl, table.double(), p, nfft, iw)           # [iw][cc][c]
        Ut = torch.empty_like(U[f:f + step])
        for s in range(ns):
            i = ti(cr[s])
            Ut[:, s] = (H[:, i[None, :], i[:, None]] * Wr @ U[f:f + step, s, :, None])[..., 0]
        out = torch.zeros_like(Ut)
        for r in range(ns + nh - 1):                                    # equal spacings: trace r - is of shot is
            lo, hi = max(0, r - (nh - 1)), min(ns - 1, r)
            if hi < lo:
                continue
            sh = np.arange(lo, hi + 1)
            i, h = ti(cs[sh]), ti(r - sh)
            W = _side(len(sh), dx, dat, ap, tap)
            v = Ut[:, ti(sh), h]
            out[:, ti(sh), h] += (H[:, i[None, :], i[:, None]] * W @ v[..., None])[..., 0]
        U[f:f + step] = out
    res = torch.empty((ns, nh, nt), dtype=F64, device="cuda")
    for s in range(0, ns, 8):
        res[s:s + 8] = torch.flip(torch.fft.irfft(U[:, s:s + 8].permute(1, 2, 0), n=nfft)[..., :nt], [-1])
    return res


def _stitch64(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rows = _rows(c)
    layers = [torch.randn((c["n3"], c["n2"], e - s + 1), generator=gen, dtype=F32, device="cuda") for s, e in rows]
    out = torch.zeros((c["n3"], c["n2"], c["n1"]), dtype=F64, device="cuda")
    i = np.arange(c["n2"])
    edge, a = np.minimum(i, c["n2"] - 1 - i), c["aper"]
    lat = torch.from_numpy(np.where(edge < a, 1.0 + 0.5 * (1.0 - edge / max(1, a - 1)), 1.0)).cuda()[None, :, None]
    prev = -1
    for k, ((s, e), v) in enumerate(zip(rows, layers)):
        v = v.double() * _stitch_scales(c)[k] * (lat if k else 1.0)
        over = prev - s + 1 if k else 0
        blend = over if c["blend"] < 0 else min(c["blend"], over)
        keep = over - blend
        out[:, :, s + over:e + 1] = v[:, :, over:]
        if blend > 0:
            u = torch.arange(blend, dtype=F64, device="cuda") / (blend - 1) if blend > 1 else torch.ones(1, dtype=F64, device="cuda")
            w = 0.5 * (1 - torch.cos(math.pi * u))
            sl = slice(s + keep, s + over)
            out[:, :, sl] = out[:, :, sl] * (1 - w) + v[:, :, keep:over] * w
        prev = e
    return out


def exact(case, seed):
    c = case
    if c["kind"] == "migrate":
        if c["ns"] * c["nh"] * c["nz"] * c["nx"] > 6e9:
            return None  # the production survey takes minutes in plain torch
        T, D = _tables(c, seed)
        ng, g0, dg = _axis(c)
        data = _gathers(_offsets(c), c["nt"], c["dt"], seed, 15.0)
        return _image64(c, seed, _survey_shots(c, ng, g0, dg), ng, g0, dg, T, D, data)
    if c["kind"] == "model":
        return _model64(c, seed)
    if c["kind"] == "windows":
        out = []
        for w in range(c["windows"]):
            cw = dict(_window(c, w), mode="angle", interp="h", cmp=0, nt=c["tmax"], nh=1, ns=1, h0=0.0, s0=0.0, ds=0.0)
            T, D = _tables(cw, seed + w)
            rec = _window_shots(c, seed, w)
            shots = [(s["sx"], np.float32(s["sx"]), [float(v) for v in s["h"]], s["h"], 0.0, f32(c["dh"]),
                      s["data"].shape[1], None, None) for s in rec]
            out.append(_image64(cw, seed, shots, 61, 0.0, 1.0, T, D, [s["data"] for s in rec]))
        return out
    if c["kind"] == "datum":
        return _datum64(c, seed)
    if c["kind"] == "stitch":
        return [_stitch64(c, seed), None]
    # a table is the fixed point of float updates in the sweeps' own order: it has no separate 64-bit value
    return None
