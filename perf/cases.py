"""Performance cases of the FWI gradient path: what a user's program runs.

A case is a dict of plain values.  ``kind`` names the call:

  gradient  Survey.set_lambda + Survey.run(1): one calculate_misfit_gradient
            over all shots (forward, misfit, adjoint, imaging, stack)
  trial     one line-search trial: Survey.set_time (the trial model's time
            axis with its resampled data), set_lambda, run(2), and the
            synthetic gather of the first shot
  batch     calculate_misfit_gradient with host buffers, as a Fortran driver
            calls it
  dropin    one shot through the drop-in routines: solver_acoustic_SS
            forward, Misfit_function, solver_acoustic_SS adjoint
  green     solver_acoustic_SS forward for an impulse, traces only, on the
            wide CPML of the source estimation
  prep      a band's trace preparation: time_filter, interpolation_akima
  nlcg      Beta_calculous, first_step and model_update of one iteration

Observed traces are hyperbolic Ricker events, models are water over layers
with a lateral perturbation; everything comes from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import fwi_gb300 as F
from fwi_gb300 import ShotSpec, SurveySpec

F32 = np.float32
SNAP = {"f32": F.SNAP_F32, "bf16": F.SNAP_BF16, "f16": F.SNAP_F16}
_stream = None


def _base(kind, **kw):
    c = dict(kind=kind, ny=200, nx=400, d=25.0, dt=0.002, nt=400, shots=1, channels=100, drec=25.0, window="full",
             acc=3, dpml=20, store_snap=10, snap="f32", recompute=False, freq=8.0)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest survey a program or a test runs: latency alone
        _base("gradient", name="tiny_gradient", ny=40, nx=90, d=10.0, dt=0.001, nt=200, shots=3, channels=20,
              drec=10.0, dpml=8, freq=25.0),
        # one plain shot, 8th order, full record
        _base("gradient", name="single_gradient", nt=3000, channels=200, drec=12.5, acc=4),
        # a small field survey on an odd grid (the example job's model size), 6th order
        _base("gradient", name="field_gradient", ny=163, nx=384, nt=1000, shots=12, channels=120),
        # the batched MCS survey: all 64 shots on the full model (the largest case)
        _base("gradient", name="mcs_gradient", ny=400, nx=2000, d=12.5, dt=0.001, nt=1200, shots=64, channels=480,
              drec=12.5, freq=10.0),
        # the precision form: FP16 snapshots every 4 steps, checkpointed recomputation
        _base("gradient", name="mcs_f16_recompute", ny=400, nx=2000, d=12.5, dt=0.001, nt=600, shots=16,
              channels=480, drec=12.5, freq=10.0, store_snap=4, snap="f16", recompute=True),
        # OBS sources on uneven windows of a crustal model
        _base("gradient", name="was_gradient", ny=600, nx=6000, dt=0.0015625, nt=800, shots=8, window="uneven",
              channels=0, drec=125.0, freq=8.0),
        # a line-search trial of the inversion workload: streamer windows, a new time axis per call
        _base("trial", name="inversion_trial", ny=600, nx=3000, d=12.5, dt=0.001, nt=640, shots=24, channels=480,
              drec=12.5, freq=10.0, window="streamer"),
        # the drop-in batch call with host buffers on ragged sizes
        _base("batch", name="host_batch", ny=251, nx=1013, d=12.5, dt=0.00125, nt=730, shots=10, channels=240,
              drec=12.5, freq=10.0),
        # one shot through the routines of the reference's shot loop
        _base("dropin", name="dropin_shot", ny=163, nx=384, nt=1000, channels=120),
        # Green's functions of the source estimation (two strip columns per lane)
        _base("green", name="source_green", ny=150, nx=301, nt=800, channels=96, dpml=50),
        # one band's data: low-pass and resampling of a survey's traces
        dict(kind="prep", name="band_traces", traces=3840, nt=2000, dt=0.002, nt_out=3130, dt_out=0.00127797,
             typef=1, f1=2.0, fc=5.0),
        # the model arithmetic of one NLCG iteration on the inversion workload's model
        dict(kind="nlcg", name="nlcg_step", ny=600, nx=3000),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["gradient"] * 6 + ["trial", "batch", "dropin", "green", "prep", "nlcg"])
    if kind == "prep":
        nt = _log(rng, 300, 4000)
        dt = rng.choice([0.002, 0.004])
        k = rng.uniform(0.6, 2.0)
        return dict(kind=kind, traces=_log(rng, 24, min(8000, 8_000_000 // nt)), nt=nt, dt=dt, nt_out=int(nt * k),
                    dt_out=dt / k, typef=rng.choice([1, 1, 3]), f1=2.0, fc=rng.choice([3.0, 5.0, 7.0]))
    if kind == "nlcg":
        return dict(kind=kind, ny=_log(rng, 40, 600), nx=_log(rng, 90, 6000))
    acc = rng.choice([3, 3, 4])
    d = rng.choice([12.5, 25.0])
    c = _base(kind, d=d, dt=d / 12500.0, acc=acc, ny=_log(rng, 40, 600), freq=10.0 if d < 20 else 8.0)
    if kind in ("dropin", "green"):
        c.update(nx=_log(rng, 90, 800), ny=min(c["ny"], 300), nt=_log(rng, 350, 1500), channels=_log(rng, 10, 200),
                 dpml=50 if kind == "green" else 20)
    else:
        c.update(window=rng.choice(["full", "full", "streamer", "uneven"]), shots=_log(rng, 1, 64),
                 snap=rng.choice(["f32", "f32", "f16", "bf16"]), recompute=rng.random() < 0.15,
                 channels=_log(rng, 20, 480))
        c["store_snap"] = rng.choice([10, 5] if c["snap"] == "f32" else [10, 4])
        c["nx"] = _log(rng, 400, 6000) if c["window"] == "uneven" else _log(rng, 90, 3000)
        c["drec"] = 125.0 if c["window"] == "uneven" else d
        if kind == "batch":
            c["recompute"] = False
    room = int((c["nx"] * d - 400.0) / c["drec"])  # the streamer lies inside the model
    c["channels"] = 0 if c["window"] == "uneven" else max(4, min(c["channels"], room))
    # no more work than the largest listed case
    per = (c["ny"] + 26) * sum(w + 52 for _, w in _windows(c)) * 2.0 * (3 if c["recompute"] else 2)
    top = min(3000, int(426 * 2052 * 64 * 1200 / per))
    if kind not in ("dropin", "green"):
        least = int((0.9 if c["window"] == "uneven" else 0.35) / c["dt"])  # the waves reach some receivers
        if top < least:
            c.update(shots=max(1, c["shots"] * top // least))
            top = least
        c["nt"] = _log(rng, least, max(least + 1, top))
    c["freq"] = max(c["freq"], 8.0 / (c["nt"] * c["dt"]))
    ss = c["store_snap"]
    c["nt"] = c["nt"] // ss * ss  # whole snapshot blocks, as the time rules give
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _source_x(c, i):
    """x (m) of shot i: evenly spread where its streamer lies inside the model."""
    length = c["nx"] * c["d"]
    lo = 150.0 + c["channels"] * c["drec"] + 2 * c["d"] if c["channels"] else 4 * c["d"]
    hi = max(lo, length - 4 * c["d"])
    return lo + (hi - lo) * ((i + 0.5) / c["shots"])


def _windows(c):
    """(first column, width) per shot: the same for every seed (a survey's geometry)."""
    out = []
    nx, d = c["nx"], c["d"]
    for i in range(c["shots"]):
        x = int(_source_x(c, i) / d)
        if c["window"] == "streamer":
            m = 160
            lo, hi = max(0, x - int((150.0 + c["channels"] * c["drec"]) / d) - m), min(nx, x + m)
        elif c["window"] == "uneven":
            w = int(nx * (0.2 + 0.47 * ((0.37 + 0.618034 * i) % 1.0)))
            lo, hi = max(0, x - w // 2), min(nx, x + w // 2 + 1)
        else:
            lo, hi = 0, nx
        out.append((lo, hi - lo))
    return out


def _ricker(t, f):
    a = (math.pi * f * t) ** 2
    return (1 - 2 * a) * np.exp(-a)


def _model(c, rng):
    """Water over eight layers with a lateral perturbation, no faster than the time step allows."""
    ny, nx, d = c["ny"], c["nx"], c["d"]
    vmax = min(5000.0, 0.5 * d / c["dt"])
    z, x = (np.arange(ny) + 0.5) * d, (np.arange(nx) + 0.5) * d
    depth = ny * d
    sea = min(0.2 * depth, 800.0)
    tops = np.sort(rng.uniform(sea, 0.95 * depth, 8))
    tops[0] = sea
    vels = np.sort(rng.uniform(1700.0, 0.93 * vmax, 8))
    vp = np.full((ny, nx), 1500.0)
    for t, v in zip(tops, vels):
        pert = 1 + 0.06 * np.sin(2 * np.pi * x / rng.uniform(2000.0, 9000.0) + rng.uniform(0, 2 * np.pi))
        vp[z >= t, :] = v * pert[None, :]
    vp = np.minimum(vp, vmax).astype(F32)
    lam = np.asfortranarray(F32(1000.0) * (vp * vp))
    return vp, lam, int(tops[0] / d)


def _observed(c, spec, rng):
    """All shots' traces packed in shot order, (traces, nt) on the device: a
    direct arrival and four reflection hyperbolas with the geometry's
    distances.  Traces that the direct wave reaches late in the record or
    after it are dead (zero), as muted far offsets are."""
    off = np.concatenate([np.hypot(s.nxRec.astype(np.float64) - s.nxSou[0], s.nyRec - s.nySou[0])
                          for s in spec.shots]) * c["d"]
    ev = [(0.0, 1500.0, 1.0)] + [(rng.uniform(0.05, 0.9) * c["nt"] * c["dt"], rng.uniform(1600.0, 3000.0),
                                  rng.uniform(0.1, 0.5)) for _ in range(4)]
    x = torch.from_numpy(off).cuda()[:, None]
    t = torch.arange(c["nt"], dtype=torch.float64, device="cuda")[None, :] * c["dt"]
    out = torch.zeros((off.size, c["nt"]), dtype=torch.float32, device="cuda")
    for t0, v, amp in ev:
        a = (math.pi * c["freq"] * (t - 1.5 / c["freq"] - torch.sqrt(t0 * t0 + (x / v) ** 2))) ** 2
        out += (amp * (1 - 2 * a) * torch.exp(-a)).float()
    out *= (x / 1500.0 + 2.0 / c["freq"] < c["nt"] * c["dt"]).float()
    return out


def _survey(c, seed):
    """(spec without observed data, velocity, lambda, observed traces on the device)."""
    rng = np.random.default_rng(seed)
    vp, lam, water = _model(c, rng)
    d, nt = c["d"], c["nt"]
    shots = []
    for i, (x0, w) in enumerate(_windows(c)):
        xs = _source_x(c, i)
        nxs = min(1 + math.ceil(xs / d), x0 + w)
        if c["channels"]:
            pos = xs - 150.0 - c["drec"] * np.arange(c["channels"])
            nxr = np.clip(1 + np.ceil(pos / d).astype(np.int32), x0 + 1, x0 + w)
        else:  # surface receivers over the whole model, those inside the window
            grid = 1 + np.ceil(np.arange(62.5, c["nx"] * d, c["drec"]) / d).astype(np.int32)
            nxr = grid[(grid > x0) & (grid <= x0 + w)]
        row = 1 + math.ceil(10.0 / d)
        shift = rng.uniform(0.0, 0.01)
        src = _ricker(np.arange(nt) * c["dt"] - 1.5 / c["freq"] - shift, c["freq"]).astype(F32)
        shots.append(ShotSpec(x0=x0, nx=w, nxSou=np.array([nxs - x0], np.int32),
                              nySou=np.array([row if c["channels"] else max(row, min(water, c["ny"] - 2))], np.int32),
                              nxRec=(nxr - x0).astype(np.int32), nyRec=np.full(nxr.size, row, np.int32),
                              src=np.asfortranarray(src.reshape(nt, 1))))
    spec = SurveySpec(ny=c["ny"], nx_model=c["nx"], d=d, dt=c["dt"], nt=nt, shots=shots, store_snap=c["store_snap"],
                      acc=c["acc"], dpml=c["dpml"], water_rows=np.full(c["nx"], min(water, c["ny"] // 4), np.int32))
    return spec, vp, lam, _observed(c, spec, rng)


def _traces(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.arange(c["nt"], dtype=torch.float32, device="cuda")[None, :] * c["dt"]
    x = torch.rand((c["traces"], 6), generator=g, device="cuda")
    out = 0.02 * torch.randn((c["traces"], c["nt"]), generator=g, device="cuda")
    for k in range(6):
        a = (math.pi * (6.0 + 2 * k) * (t - x[:, k:k + 1] * c["nt"] * c["dt"])) ** 2
        out += (1 - 2 * a) * torch.exp(-a) / (k + 1)
    return out.contiguous()


def _nlcg(c, seed):
    rng = np.random.default_rng(seed)
    shape = (c["ny"], c["nx"])
    z = np.linspace(0, 1, c["ny"])[:, None]
    old = rng.standard_normal(shape) * np.exp(-2 * z) * 1e-9
    grad = 0.5 * old + rng.standard_normal(shape) * np.exp(-2 * z) * 5e-10
    var = 1000.0 * (1500.0 + 3000.0 * z + 100.0 * rng.random(shape)) ** 2
    return [np.asfortranarray(a.astype(F32)) for a in (grad, old, var)]


def _on_stream():
    """One torch stream for the program's own work and the library's."""
    global _stream
    if _stream is None:
        F.init(0)
        _stream = torch.cuda.Stream()
        F.set_stream(_stream.cuda_stream)
    return torch.cuda.stream(_stream)


def prepare(case, seed):
    c = case
    with _on_stream():
        if c["kind"] == "prep":
            raw = _traces(c, seed)
            return dict(c=c, raw=raw, work=torch.empty_like(raw))
        if c["kind"] == "nlcg":
            grad, old, var = _nlcg(c, seed)
            return dict(c=c, grad=grad, old=old, var=var, search=np.asfortranarray(-grad))
        spec, vp, lam, obs = _survey(c, seed)
        s = dict(c=c, spec=spec, lam=lam, obs=obs)
        if c["kind"] in ("gradient", "trial"):
            s["sv"] = F.Survey(spec, snap_form=SNAP[c["snap"]], recompute=c["recompute"])
            s["sv"].set_observed(obs.data_ptr())
            s["grad"] = np.zeros((c["ny"], c["nx"]), F32, order="F")
            s["src"] = torch.from_numpy(np.concatenate([sh.src.reshape(-1) for sh in spec.shots])).cuda()
        elif c["kind"] == "batch":
            host, at = obs.cpu().numpy(), 0
            for sh in spec.shots:
                n = len(sh.nxRec)
                sh.obs = host[at:at + n].T
                at += n
            s["grad"] = np.zeros((c["ny"], c["nx"]), F32, order="F")
        else:
            ny, nx, nt, n = c["ny"], c["nx"], c["nt"], c["channels"]
            s["vp"] = np.asfortranarray(vp)
            s["rec"] = np.zeros((nt, n), F32, order="F")
            if c["kind"] == "green":
                s["S"] = np.zeros((nt, 1), F32, order="F")
                s["S"][0, 0] = F32(1.0) / F32(c["dt"])
            else:
                s["S"] = spec.shots[0].src
                s["trace"] = np.asfortranarray(obs.cpu().numpy().T)
                s["fields"] = np.zeros((ny, nx * (nt // c["store_snap"] + 1)), F32, order="F")
                s["kernel"] = np.zeros((ny, nx), F32, order="F")
                s["adj"] = np.zeros((nt, n), F32, order="F")
                s["rec2"] = np.zeros((nt, n), F32, order="F")
        _stream.synchronize()
    return s


def run(s):
    c = s["c"]
    with _on_stream():
        return _RUN[c["kind"]](s, c)


def _run_gradient(s, c):
    s["grad"][...] = 0.0
    s["sv"].set_lambda(s["lam"])
    misfit, grad = s["sv"].run(1, s["grad"])
    return dict(misfit=misfit, grad=grad)


def _run_trial(s, c):
    sv = s["sv"]
    sv.set_time(c["dt"], c["nt"], s["src"].data_ptr(), s["obs"].data_ptr())
    sv.set_lambda(s["lam"])
    misfit, _ = sv.run(2)
    return dict(misfit=misfit, synthetic=sv.synthetic(0))


def _run_batch(s, c):
    s["grad"][...] = 0.0
    misfit = F.calculate_misfit_gradient(s["spec"], s["lam"], 1, 0.0, s["grad"], snap_form=SNAP[c["snap"]])
    return dict(misfit=misfit, grad=s["grad"])


def _run_dropin(s, c):
    sh = s["spec"].shots[0]
    ny, nx, nt, n, ss = c["ny"], c["nx"], c["nt"], c["channels"], c["store_snap"]
    F.set_solver_options(c["acc"], c["dpml"])
    geo = (sh.nxSou, sh.nySou, sh.nxRec, sh.nyRec)
    F.solver_acoustic_SS(0, 1, 1, n, *geo, s["S"], None, c["d"], c["dt"], ny, nx, s["vp"], ss, nt // ss, nt,
                         s["kernel"], s["fields"], s["rec"])
    misfit, _ = F.Misfit_function(0, c["freq"], s["rec"], s["trace"], n, nt, c["dt"], s["adj"])
    s["kernel"][...] = 0.0
    F.solver_acoustic_SS(0, 2, 1, n, *geo, s["S"], s["adj"], c["d"], c["dt"], ny, nx, s["vp"], ss, nt // ss, nt,
                         s["kernel"], s["fields"], s["rec2"])
    return dict(rec=s["rec"], fields=s["fields"], misfit=misfit, adj=s["adj"], kernel=s["kernel"])


def _run_green(s, c):
    sh = s["spec"].shots[0]
    F.set_solver_options(c["acc"], c["dpml"])
    F.solver_acoustic_SS(0, 0, 1, c["channels"], sh.nxSou, sh.nySou, sh.nxRec, sh.nyRec, s["S"], None, c["d"],
                         c["dt"], c["ny"], c["nx"], s["vp"], c["nt"] + 1, 0, c["nt"], None, None, s["rec"])
    return s["rec"]


def _run_prep(s, c):
    s["work"].copy_(s["raw"])
    F.time_filter(s["work"].data_ptr(), c["nt"], c["dt"], c["traces"], c["typef"], c["f1"], c["fc"])
    out = torch.empty((c["traces"], c["nt_out"]), dtype=torch.float32, device="cuda")
    F.interpolation_akima(s["work"].data_ptr(), c["dt"], c["nt"], c["traces"], c["dt_out"], c["nt_out"],
                          out=out.data_ptr())
    return dict(filtered=s["work"], resampled=out)


def _run_nlcg(s, c):
    beta, num, den = F.Beta_calculous(s["grad"], s["old"], c["nx"], c["ny"])
    nut = F.first_step(s["search"], s["var"])
    return dict(beta=beta, num=num, den=den, nut=nut, lam=F.model_update(s["search"], s["var"], nut))


_RUN = dict(gradient=_run_gradient, trial=_run_trial, batch=_run_batch, dropin=_run_dropin, green=_run_green,
            prep=_run_prep, nlcg=_run_nlcg)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    """Every array of a pass read and written once: a time step reads p, p_1 and
    c2 and writes p_3 of every cell below the free surface and reads and writes
    two memory variables of every CPML cell; a gradient stores and reads its
    snapshots and updates its accumulator.  Operations: one rounded multiply
    or add each."""
    c = case
    if c["kind"] == "prep":
        n = c["traces"]
        ts = 24 * c["nt"]
        return dict(bytes=4.0 * n * (2 * c["nt"] + c["nt_out"]),
                    flops=n * (5.0 * ts * math.log2(ts) + 3 * ts + 60 * c["nt_out"]))
    if c["kind"] == "nlcg":
        n = c["ny"] * c["nx"]
        return dict(bytes=4.0 * n * 5, flops=40.0 * n)
    dn = c["dpml"] + 2 * c["acc"]
    passes = {"gradient": 2, "batch": 2, "dropin": 2, "trial": 1, "green": 1}[c["kind"]]
    if c["recompute"]:
        passes = 3
    b = f = 0.0
    for _, w in _windows(c):
        cells = (c["ny"] + dn) * (w + 2.0 * dn)
        pml = 2.0 * c["ny"] * dn + dn * w + 4.0 * dn * dn
        b += c["nt"] * passes * 16.0 * (cells + pml)
        f += c["nt"] * passes * ((6 * c["acc"] + 9) * cells + (6 * c["acc"] + 10) * pml)
        if passes > 1:
            es = 4 if c["snap"] == "f32" else 2
            b += (c["nt"] // c["store_snap"]) * c["ny"] * w * ((2 if passes == 2 else 3) * es + 8.0)
            f += (c["nt"] // c["store_snap"]) * c["ny"] * w * 7.0
    return dict(bytes=b, flops=f)


# ---------------------------------------------------------------------------
# the same results in 64 bits: plain torch
# ---------------------------------------------------------------------------

_C1 = {3: [3 / 4, -3 / 20, 1 / 60], 4: [4 / 5, -1 / 5, 4 / 105, -1 / 280]}
_C2 = {3: [-49 / 18, 3 / 2, -3 / 20, 1 / 90], 4: [-205 / 72, 8 / 5, -1 / 5, 8 / 315, -1 / 560]}


def _clamped(f, dim, R, taps, even):
    """Central difference along dim of f; the R values at either end copy the nearest inner one."""
    n = f.shape[dim]
    mid = lambda o: f.narrow(dim, R + o, n - 2 * R)  # noqa: E731
    out = taps[0] * mid(0) if even else 0
    for i in range(1, R + 1):
        t = taps[i] if even else taps[i - 1]
        out = out + t * (mid(i) + mid(-i) if even else mid(i) - mid(-i))
    lo, hi = out.narrow(dim, 0, 1), out.narrow(dim, n - 2 * R - 1, 1)
    shape = list(f.shape)
    shape[dim] = R
    return torch.cat([lo.expand(shape), out, hi.expand(shape)], dim)


class _Wave:
    """Acoustic propagation of shots of one window width, (shots, rows, columns)
    below the free surface, CPML on the sides and at the bottom."""

    def __init__(self, c, vp):
        R, dn = c["acc"], c["dpml"] + 2 * c["acc"]
        self.R, self.dn, self.c = R, dn, c
        self.S, self.ny, self.nx = vp.shape
        d, dt = float(F32(c["d"])), float(F32(c["dt"]))
        v = torch.cat([vp[:, :, :1].expand(-1, -1, dn), vp, vp[:, :, -1:].expand(-1, -1, dn)], 2)
        v = torch.cat([v, v[:, -1:, :].expand(-1, dn, -1)], 1)
        self.c2 = v * v * (dt * dt) / (d * d)
        i = np.arange(c["dpml"]) * d
        w = (c["dpml"] - 1) * d
        alpha = 30 * math.pi * (1 - i / w)
        sigma = -((6000.0 * math.log(1e-5)) / (2 * w)) * (i / w) ** 2
        a = np.exp(-(sigma + alpha) * dt)
        A = np.concatenate([np.zeros(R), a, np.full(R, a[-1])])
        b = (a - 1) * sigma / np.maximum(sigma + alpha, 1e-300)
        B = np.concatenate([np.zeros(R), b, np.full(R, b[-1])])
        rows = np.concatenate([np.full(self.ny, -1), np.arange(dn)])
        right = np.maximum(rows[:, None], np.arange(dn)[None, :])
        left = np.maximum(rows[:, None], np.arange(dn)[::-1][None, :])
        cols = np.concatenate([np.arange(dn)[::-1], np.full(self.nx, -1), np.arange(dn)])
        bot = np.maximum(np.arange(dn)[:, None], cols[None, :])
        g = lambda t, ix: torch.from_numpy(t[ix]).cuda()  # noqa: E731
        self.f = [(g(A, ix), g(B, ix)) for ix in (left, right, bot)]
        self.zero()

    def zero(self):
        z = lambda *s: torch.zeros(s, dtype=torch.float64, device="cuda")  # noqa: E731
        h, w, dn = self.ny + self.dn, self.nx + 2 * self.dn, self.dn
        self.p, self.p1 = z(self.S, h, w), z(self.S, h, w)
        self.phi = [z(self.S, h, dn), z(self.S, h, dn), z(self.S, dn, w)]
        self.chi = [t.clone() for t in self.phi]

    def step(self, cells, values):
        """One time step; cells = (shot, row, column) index tensors, values injected there."""
        R, dn, p = self.R, self.dn, self.p
        c1, c2 = _C1[R], _C2[R]
        top = torch.cat([torch.zeros_like(p[:, :R]), p], 1)  # the free surface reads zero above
        d2x = _clamped(p, 2, R, c2, True)
        d2y = _clamped(top, 1, R, c2, True)[:, R:]
        tot = d2x + d2y
        strips = [(2, slice(None), slice(0, dn)), (2, slice(None), slice(self.nx + dn, None)),
                  (1, slice(self.ny, None), slice(None))]
        dx = [_clamped(p[:, :, :dn + 2 * R], 2, R, c1, False)[:, :, :dn],
              _clamped(p[:, :, self.nx + dn - 2 * R:], 2, R, c1, False)[:, :, 2 * R:],
              _clamped(p[:, self.ny - 2 * R:], 1, R, c1, False)[:, 2 * R:] if self.ny >= 2 * R else
              _clamped(top, 1, R, c1, False)[:, R + self.ny:]]
        for k, (dim, rs, cs) in enumerate(strips):
            A, B = self.f[k]
            dphi = _clamped(self.phi[k], dim, R, c1, False)
            d2 = (d2x if dim == 2 else d2y)[:, rs, cs]
            self.phi[k] = A * self.phi[k] + B * dx[k]
            self.chi[k] = A * self.chi[k] + B * (d2 + dphi)
            tot[:, rs, cs] += dphi + self.chi[k]
        if cells is not None:
            tot.index_put_(cells, values, accumulate=True)
        p3 = 2 * p - self.p1 + self.c2 * tot
        old = self.p1
        self.p1, self.p = p, p3
        return p3, old


def _cells(shots, ny, nx, dn, which):
    """Injection cells (shot, row, column) and value index: interior cells, the last of each cell."""
    last = {}
    at = 0
    for s, sh in enumerate(shots):
        xs, ys = (sh.nxSou, sh.nySou) if which == "sou" else (sh.nxRec, sh.nyRec)
        for j in range(len(xs)):
            if 1 <= xs[j] <= nx and 1 <= ys[j] <= ny:
                last[(s, int(ys[j]) - 1, int(xs[j]) - 1 + dn)] = at + j
        at += len(xs)
    t = lambda v: torch.tensor(v, dtype=torch.long, device="cuda")  # noqa: E731
    keys = list(last)
    return tuple(t([k[i] for k in keys]) for i in range(3)), t([last[k] for k in keys])


def _gradient64(c, shots, vp, src, obs, adjoint=True, keep=False):
    """Shots of one width: (misfit, kernels (shots, ny, nx), traces, snapshots, adjoint sources)."""
    w = _Wave(c, vp)
    ny, nx, dn, nt, ss = w.ny, w.nx, w.dn, c["nt"], c["store_snap"]
    dt = float(F32(c["dt"]))
    cells, ix = _cells(shots, ny, nx, dn, "sou")
    n = [len(sh.nxRec) for sh in shots]
    cat = lambda a: torch.from_numpy(np.concatenate(a).astype(np.int64)).cuda()  # noqa: E731
    rs = torch.repeat_interleave(torch.arange(len(shots)).cuda(), torch.tensor(n).cuda())
    ry, rx = cat([sh.nyRec for sh in shots]) - 1, cat([sh.nxRec for sh in shots]) - 1 + dn
    rec = torch.zeros((sum(n), nt), dtype=torch.float64, device="cuda")
    snaps = [torch.zeros((len(shots), ny, nx), dtype=torch.float64, device="cuda")]
    lap = 1
    for k in range(2, nt + 1):
        p3, old = w.step(cells, src[ix, k - 2])
        rec[:, k - 2] = p3[rs, ry, rx]
        lap += 1
        if lap == ss:
            lap = 0
            if adjoint:
                snaps.append((p3 - old)[:, :ny, dn:dn + nx] * 0.5 / dt)
    rec[:, nt - 1] = rec[:, nt - 2]
    if obs is None:
        return 0.0, None, rec, None, None
    ms, mt = rec.abs().amax(1, keepdim=True), obs.abs().amax(1, keepdim=True)
    use = (ms > 0) & (mt > 0)
    r = torch.where(use, rec / ms.clamp_min(1e-300) - obs / mt.clamp_min(1e-300), torch.zeros_like(rec))
    misfit = float((0.5 * dt * r * r).sum())
    if not adjoint:
        return misfit, None, rec, None, None
    adj = -r.flip(1)
    cells, ix = _cells(shots, ny, nx, dn, "rec")
    w.zero()
    kern = torch.zeros_like(snaps[0])
    blk, lap = nt // ss, 1
    for k in range(2, nt + 1):
        p3, old = w.step(cells, adj[ix, k - 2])
        lap += 1
        if lap == ss:
            lap = 0
            blk -= 1
            kern -= 0.5 * (p3 - old)[:, :ny, dn:dn + nx] * snaps[blk] * ss
    return misfit, kern, rec, snaps if keep else None, adj


def _cost64(c):
    """Seconds of _gradient64, roughly: launches, and about 1 KB moved per cell and step."""
    widths = sorted(w for _, w in _windows(c))
    passes = 1 if c["kind"] in ("trial", "green") else 2
    cells = (c["ny"] + 26) * sum(w + 52.0 for w in widths)
    return passes * c["nt"] * (len(set(widths)) * 6e-4 + cells * 2.0e-10)


def exact(case, seed):
    c = case
    if c["kind"] == "nlcg":
        grad, old, var = (a.astype(np.float64) for a in _nlcg(c, seed))
        num, den = float((grad * (grad - old)).sum()), float((old * old).sum())
        nut = 0.01 / np.abs(-grad / np.log(var)).max()
        return dict(beta=num / den, num=num, den=den, nut=nut, lam=np.exp(-grad * nut) * var)
    if c["kind"] == "prep":
        return _prep64(c, _traces(c, seed).double())
    if _cost64(c) > 12.0:
        return None
    spec, vp, lam, obs = _survey(c, seed)
    if c["kind"] == "dropin":
        vp64 = torch.from_numpy(vp).cuda().double()[None]
    else:
        vp64 = torch.sqrt(torch.from_numpy(np.ascontiguousarray(lam)).cuda().double() / 1000.0)[None]
    obs = obs.double()
    if c["kind"] in ("dropin", "green"):
        src = torch.from_numpy(spec.shots[0].src.T.copy()).cuda().double()
        if c["kind"] == "green":
            src = torch.zeros_like(src)
            src[0, 0] = 1.0 / float(F32(c["dt"]))
            vp64 = torch.from_numpy(vp).cuda().double()[None]
            return _gradient64(c, spec.shots, vp64, src, None, adjoint=False)[2].T
        m, kern, rec, snaps, adj = _gradient64(c, spec.shots, vp64, src, obs, keep=True)
        fields = torch.cat([s[0] for s in snaps], 1)
        return dict(rec=rec.T, fields=fields, misfit=m, adj=adj.T, kernel=kern[0])
    misfit, grad = 0.0, torch.zeros((c["ny"], c["nx"]), dtype=torch.float64, device="cuda")
    first = None
    at = np.concatenate([[0], np.cumsum([len(sh.nxRec) for sh in spec.shots])])
    for width in sorted({sh.nx for sh in spec.shots}):
        ids = [i for i, sh in enumerate(spec.shots) if sh.nx == width]
        sh = [spec.shots[i] for i in ids]
        v = torch.cat([vp64[:, :, s.x0:s.x0 + s.nx] for s in sh])
        src = torch.from_numpy(np.stack([s.src[:, 0] for s in sh])).cuda().double()
        o = torch.cat([obs[at[i]:at[i + 1]] for i in ids])
        m, kern, rec, _, _ = _gradient64(c, sh, v, src, o, adjoint=c["kind"] != "trial")
        misfit += m
        if 0 in ids:
            lo = sum(len(spec.shots[i].nxRec) for i in ids[:ids.index(0)])
            first = rec[lo:lo + len(spec.shots[0].nxRec)].T
        if kern is not None:
            for s, k in zip(sh, kern):
                grad[:, s.x0:s.x0 + s.nx] += k
    if c["kind"] == "trial":
        return dict(misfit=misfit, synthetic=first)
    grad[:int(spec.water_rows[0])] = 0.0
    return dict(misfit=misfit, grad=grad)


def _prep64(c, x):
    """Butterworth response (order 6) on the 24-fold padded traces, then Akima's cubic at the new samples."""
    nt, n = c["nt"], 6
    ts = 24 * nt
    f = torch.arange(ts // 2 + 1, dtype=torch.float64, device="cuda") / (ts * float(F32(c["dt"])))
    H = torch.ones_like(f, dtype=torch.complex128)
    f1, fc = c["f1"], c["fc"]
    f0, q = math.sqrt(f1 * fc), math.sqrt(f1 * fc) / (fc - f1)
    for k in range(1, n // 2 + 1):
        a = math.cos((2 * k + n - 1) * math.pi / (2 * n))
        s = 1j * f / fc if c["typef"] == 1 else q * (1j * f / f0 + f0 / (1j * f.clamp_min(1e-300)))
        H = H / (s * s - 2 * s * a + 1)
    H[0] = 1.0 if c["typef"] == 1 else 0.0
    H[-1] = complex(float(H[-1].real), 0.0)
    y = torch.empty_like(x)
    for i in range(0, x.shape[0], 512):
        buf = torch.zeros((x[i:i + 512].shape[0], ts), dtype=torch.float64, device="cuda")
        buf[:, ts - nt:] = x[i:i + 512]
        y[i:i + 512] = torch.fft.irfft(torch.fft.rfft(buf) * H, n=ts)[:, ts - nt:]
    return dict(filtered=y, resampled=_akima64(y, float(F32(c["dt"])), float(F32(c["dt_out"])), c["nt_out"]))


def _akima64(y, h, h_out, n_out):
    L = y.shape[1]
    m = (y[:, 1:] - y[:, :-1]) / h
    e0, e1 = 2 * m[:, :1] - m[:, 1:2], 2 * m[:, -1:] - m[:, -2:-1]
    m = torch.cat([2 * e0 - m[:, :1], e0, m, e1, 2 * e1 - m[:, -1:]], 1)  # slopes, two more at either end
    w1, w2 = (m[:, 3:] - m[:, 2:-1]).abs(), (m[:, 1:-2] - m[:, :-3]).abs()
    sw = w1 + w2
    t = torch.where(sw > 0, (w1 * m[:, 1:-2] + w2 * m[:, 2:-1]) / sw.clamp_min(1e-300),
                    0.5 * (m[:, 1:-2] + m[:, 2:-1]))
    u = torch.arange(n_out, dtype=torch.float64, device=y.device) * h_out
    i = (u / h).floor().long().clamp(0, L - 2)
    inside = u < (L - 1) * h
    s = u - i * h
    a, t3, t4, m3 = y[:, i], t[:, i], t[:, i + 1], m[:, i + 2]
    q2, q3 = (2 * (m3 - t3) + m3 - t4) / h, (t3 + t4 - 2 * m3) / (h * h)
    v = a + s * (t3 + s * (q2 + s * q3))
    # beyond the last sample: the last interval's cubic shifted outward, with equal steps
    b, tl = y[:, -1:], t[:, -1:]
    tr = 0.5 * (m[:, L + 1:L + 2] + m[:, L + 2:L + 3])
    ml, s = m[:, L + 1:L + 2], u - (L - 1) * h
    q2, q3 = (2 * (ml - tl) + ml - tr) / h, (tl + tr - 2 * ml) / (h * h)
    return torch.where(inside, v, b + s * (tl + s * (q2 + s * q3)))
