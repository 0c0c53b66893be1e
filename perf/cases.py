"""The work this package is measured on, through its public entry points.

Each case is one thing a seismic-inversion program has the engine do: one
shot at a time through the reference-shaped calls, a whole iteration's shots
in one batch, forward modelling, the line searches, Hessian products, several
models in one run, and the optimal-transport misfit by itself.  The grids,
spacings, PML widths, time steps and wavelets are those of the benchmark's
workloads, the serving stream and the tests; the number of time steps is cut
where a full-length pass would take seconds (the work per step is the same).

  shot_small       one stage-1 shot on a small grid (a test-sized survey, L2)
  shot_376         one stage-1 shot at 376x201, vertical force, OT, full nt
  shots_in_turn    the reference driver's loop: stage-2 shots one after the
                   other on one engine, each with its own window and source
  iteration_38     38 stage-2 shots at 376x201, Born + OT, Vp/Vs/rho gradients
  salt_uneven      stage-2 batch at 401x301, 12.5 m, apertures 150-401 nodes
  snapshots_2001   stage-2 shots at 2001x801 with FP16 snapshots every 4th step
  strips_on_host   a batch whose edge strips live in host memory
  model_records    forward modelling of a survey and its records
  parabola_search  the stage-1 line search: every shot at three trial models
  hessian_product  a Gauss-Newton Hessian-vector product
  several_models   requests on grids of their own and lengths of their own in one run
  ot_gathers       the OT misfit of a survey's gathers in device memory
"""
import ctypes as C
import math
import random

import numpy as np
import torch

import sfwi_gb300 as sg
from sfwi_gb300 import _lib, synth

# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # the smallest gradient call: an odd little grid where launches and latency are everything
        dict(name="shot_small", do="turn", stage=1, nx=149, nz=83, pml=11, dx=10.0, dt=1e-3, f0=25.0, nt=300, shots=1,
             misfit="l2"),
        # one full-length shot, as a program that handles one shot per call has it
        dict(name="shot_376", do="turn", stage=1, nx=376, nz=201, pml=20, dx=10.0, dt=1e-3, f0=15.0, nt=3000, shots=1,
             misfit="ot", source="vz"),
        # the drivers' loop over shots: every call brings another window, source and records
        dict(name="shots_in_turn", do="turn", stage=2, nx=299, nz=151, pml=20, dx=10.0, dt=1e-3, f0=15.0, nt=700,
             shots=4, misfit="l2", wmin=160, wmax=160),
        # one inversion iteration of the 376x201 survey
        dict(name="iteration_38", do="batch", stage=2, nx=376, nz=201, pml=20, dx=10.0, dt=1e-3, f0=15.0, nt=1000,
             shots=38, misfit="ot", rho=True),
        # uneven apertures over salt
        dict(name="salt_uneven", do="batch", stage=2, nx=401, nz=301, pml=20, dx=12.5, dt=1e-3, f0=15.0, nt=800,
             shots=20, misfit="l2", salt=True, wmin=150, wmax=401),
        # large grid, compressed snapshots instead of the reconstruction
        dict(name="snapshots_2001", do="batch", stage=2, nx=2001, nz=801, pml=20, dx=5.0, dt=5e-4, f0=25.0, nt=240,
             shots=2, misfit="ot", snap=4, fmt="f16"),
        # more strips than the device should hold: a ring of chunks, the rest in host memory
        dict(name="strips_on_host", do="batch", stage=1, nx=376, nz=201, pml=20, dx=10.0, dt=1e-3, f0=15.0, nt=700,
             shots=9, misfit="l2", ntt=50),
        # observed or synthetic data of a survey
        dict(name="model_records", do="forward", stage=1, nx=401, nz=301, pml=20, dx=12.5, dt=1e-3, f0=15.0, nt=600,
             shots=12),
        # a step length: all shots at three trial models
        dict(name="parabola_search", do="search", stage=1, nx=376, nz=201, pml=20, dx=10.0, dt=1e-3, f0=15.0, nt=600,
             shots=6, misfit="l2"),
        # a second-order step
        dict(name="hessian_product", do="hessian", stage=2, nx=251, nz=121, pml=20, dx=10.0, dt=1e-3, f0=15.0, nt=500,
             shots=5),
        # what a server runs together
        dict(name="several_models", do="models", stage=1, nx=521, nz=300, pml=20, dx=10.0, dt=1e-3, f0=15.0, nt=600,
             shots=7, models=4),
        # the misfit alone, for a program with its own propagator
        dict(name="ot_gathers", do="ot", traces=3760, nt=3000, dt=1e-3, f0=15.0, kind=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# cell-steps of a gradient pass of the largest listed case (38 x 416 x 241 x 1000)
_MOST = 38 * 416 * 241 * 1000


def draw(rng):
    do = rng.choice(["turn", "turn", "batch", "batch", "batch", "forward", "search", "hessian", "models", "ot"])
    if do == "ot":
        nt = _log(rng, 120, 7000)
        return dict(do="ot", traces=max(1, min(8000, _log(rng, 1, 12_000_000 // nt))), nt=nt, dt=1e-3, f0=15.0,
                    kind=rng.choice([1, 1, 2, 3]))
    big = rng.random() < 0.25
    pml = rng.choice([10, 11, 15, 20, 20, 20])
    dx = rng.choice([10.0, 10.0, 12.5])
    c = dict(do=do, stage=1, nx=_log(rng, 60, 1400 if big else 480), nz=_log(rng, 40, 800 if big else 320), pml=pml,
             dx=dx, dt=1e-3, f0=15.0, nt=_log(rng, 150, 1500))
    c["stage"] = 2 if do == "hessian" else 1 if do in ("search", "models") else rng.choice([1, 2])
    c["shots"] = _log(rng, 1, 4 if do == "turn" else 8 if do in ("hessian", "models") else 40)
    if do in ("turn", "batch"):
        c["misfit"] = rng.choice(["l2", "ot", "ot", "ot_power", "ot_alltrace"])
        if rng.random() < 0.4 and c["nx"] >= 120:
            c["wmin"], c["wmax"] = c["nx"] // 3, c["nx"]
            if do == "turn":
                c["wmin"] = c["wmax"] = c["nx"] // 2
        if c["stage"] == 1 and rng.random() < 0.3:
            c["source"] = "vz"
    if do == "batch":
        o = rng.choice(["plain", "plain", "rho", "snap", "host"])
        if o == "rho":
            c["rho"] = True
        elif o == "snap":
            c["snap"], c["fmt"] = rng.choice([1, 2, 4]), rng.choice(["f32", "f16", "bf16"])
        elif o == "host":
            c["ntt"] = rng.choice([20, 50, 100])
    if do == "search":
        c["misfit"] = "l2"
    if do == "models":
        c["models"] = rng.randint(1, 4)
    # no dearer than the largest listed case; a Hessian product keeps every step's velocities
    most = _MOST / (8 if do in ("hessian", "search") else 2)
    cells = lambda: (c["nx"] + 2 * pml) * (c["nz"] + 2 * pml)  # noqa: E731
    while c["shots"] * cells() * c["nt"] > most:
        c["shots"], c["nt"] = max(1, c["shots"] // 2), max(150, c["nt"] * 3 // 4)
        if c["shots"] == 1 and c["nt"] == 150:
            c["nx"], c["nz"] = c["nx"] * 3 // 4, c["nz"] * 3 // 4
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_KINDS = {"l2": sg.MISFIT_L2, "ot": sg.MISFIT_OT, "ot_power": sg.MISFIT_OT_POWER, "ot_alltrace": sg.MISFIT_OT_ALLTRACE}


def _models(case, seed, nx, nz):
    """True and starting model: layered with anomalies (or salt), and its z-smoothed form."""
    make = synth.salt_model if case.get("salt") else synth.layered_model
    vp, vs, rho = make(nx, nz, case["dx"], seed=seed, anom_seed=seed + 7)
    vp0 = synth.smooth_z(vp, 10)
    vs0 = (vp0 / 1.73).astype(np.float32)
    rho0 = (310.0 * vp0.astype(np.float64) ** 0.25).astype(np.float32)
    return dict(vp=vp, vs=vs, rho=rho, vp0=vp0, vs0=vs0, rho0=rho0, dvp=(vp - vp0).astype(np.float32),
                dvs=(vs - vs0).astype(np.float32))


def _shots(case, nx, n, seed):
    ap = (case["wmin"], case["wmax"]) if "wmin" in case else None
    return synth.config_shots(nx, case["dx"], case["pml"], n, max(1, (nx - 1) // n), aperture=ap, seed=seed)


def _engine(case, stage, nx, nz, width, nt, ntr):
    pml, dx = case["pml"], case["dx"]
    return sg.FD2DGPU_ELASTIC(synth.ricker(nt, case["dt"], case["f0"]), dx, dx, case["dt"], width + 2 * pml,
                              nz + 2 * pml, nx, nz, 1, pml, nt, 4, ntr, stage=stage)


def _source(case, fd):
    if case.get("source") == "vz":
        fd.set_source(sg.SOURCE_VZ_FORCE)


def _enqueue(case, fd, d, z=None, x=None, nt=None):
    pml = case["pml"]
    fd.enqueue_shot(d["nx"], d["isx"], pml + 2, pml, d["ngx_left"], d["delta_left"], 0, d["gc"], z, x, nt=nt)


def _pinned(a):
    p = sg.PinnedArray(a.shape)
    p.array[...] = a
    return p


def _observed(case, m, shots, nx, nz, nt):
    """Records of the true model (stage-1 modelling), in page-locked memory."""
    fd = _engine(case, 1, nx, nz, max(d["nx"] for d in shots), nt, shots[0]["ntr"])
    fd.GPUbufferVPVS(m["vp"], m["vs"], m["rho"])
    _source(case, fd)
    for d in shots:
        _enqueue(case, fd, d)
    fd.run_forward()
    out = []
    for i, d in enumerate(shots):
        r = fd.read_records(i, ntr=d["ntr"])
        out.append((_pinned(r["syn_z"]), _pinned(r["syn_x"])))
    fd.close()
    return out


def _gathers(case, seed):
    """Observed and predicted gathers on the GPU: a few wavelets with
    hyperbolic moveout per trace, the prediction shifted and scaled, and
    weak noise."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, nt, dt, f0 = case["traces"], case["nt"], case["dt"], case["f0"]
    t = torch.arange(nt, device="cuda", dtype=torch.float32) * dt
    r = lambda *s: torch.rand(*s, generator=g, device="cuda")  # noqa: E731
    off = torch.linspace(-1.0, 1.0, n, device="cuda")[:, None]
    out = {}
    for comp in ("z", "x"):
        obs = 2e-4 * (r(n, nt) - 0.5)
        cal = torch.zeros(n, nt, device="cuda")
        for _ in range(5):
            t0, v, a, s = (float(x) for x in r(4))
            arr = torch.sqrt((0.1 + 0.7 * t0) ** 2 + (off * (0.2 + v)) ** 2) * nt * dt
            for dst, shift, scale in ((obs, 0.0, 1.0), (cal, 0.02 * (s - 0.5) * nt * dt, 0.8 + 0.4 * s)):
                u = (math.pi * f0 * (t - arr - shift)) ** 2
                dst += (a - 0.5) * scale * (1 - 2 * u) * torch.exp(-u)
        out["obs_" + comp], out["cal_" + comp] = obs.contiguous(), cal.contiguous()
    return out


def _inputs(case, seed):
    """Host data of a case: models, shots, wavelet, observed records."""
    do = case["do"]
    nx, nz, nt = case["nx"], case["nz"], case["nt"]
    if do == "models":
        rng = random.Random(seed * 31 + 5)
        geo = random.Random(case["nx"] * 977 + case["nz"])  # the requests' grids belong to the case
        parts = []
        for k in range(case["models"]):
            mx, mz = nx, nz
            mt = nt
            if k:
                mx, mz, mt = (max(40, int(v * geo.uniform(0.45, 1.0))) for v in (nx, nz, nt))
            n = max(1, case["shots"] // case["models"])
            m = _models(case, rng.randrange(1 << 20), mx, mz)
            shots = synth.config_shots(mx, case["dx"], case["pml"], n, max(1, (mx - 1) // n))
            parts.append(dict(m=m, shots=shots, nx=mx, nz=mz, nt=mt, obs=_observed(case, m, shots, mx, mz, mt)))
        return dict(parts=parts)
    m = _models(case, seed, nx, nz)
    shots = _shots(case, nx, case["shots"], 3)
    obs = None if do in ("forward", "hessian") else _observed(case, m, shots, nx, nz, nt)
    return dict(m=m, shots=shots, obs=obs)


def prepare(case, seed):
    if case["do"] == "ot":
        s = _gathers(case, seed)
        s["res_z"], s["res_x"] = torch.empty_like(s["obs_z"]), torch.empty_like(s["obs_x"])
        return dict(case=case, **s)
    s = _inputs(case, seed)
    s["case"] = case
    do, nx, nz, nt, stage = case["do"], case["nx"], case["nz"], case["nt"], case["stage"]
    if do == "models":
        allsh = [d for p in s["parts"] for d in p["shots"]]
        fd = _engine(case, stage, nx, nz, max(d["nx"] for d in allsh), nt, allsh[0]["ntr"])
        fd.set_misfit(sg.MISFIT_L2)
    else:
        m, shots = s["m"], s["shots"]
        fd = _engine(case, stage, nx, nz, max(d["nx"] for d in shots), nt, shots[0]["ntr"])
        if stage == 2:
            fd.GPUbufferVPVS(m["vp0"], m["vs0"])
            fd.GPUbufferM(m["dvp"], m["dvs"])
        elif do == "forward":
            fd.GPUbufferVPVS(m["vp"], m["vs"], m["rho"])
        else:
            fd.GPUbufferVPVS(m["vp0"], m["vs0"], m["rho0"])
        fd.set_misfit(_KINDS[case.get("misfit", "l2")])
        if case.get("rho"):
            fd.set_density_gradient(True)
        if case.get("snap"):
            fd.set_snapshots(case["snap"], case["fmt"])
        if case.get("ntt"):
            fd.set_cpu_mem(True, case["ntt"])
        _source(case, fd)
    s["fd"] = fd
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------


def run(s):
    case = s["case"]
    do = case["do"]
    if do == "ot":
        n, nt = s["obs_z"].shape
        w = C.c_double(0.0)
        _lib.check(_lib.load().sfwi_ot_noalloc(
            case["kind"], s["obs_x"].data_ptr(), s["obs_z"].data_ptr(), s["cal_x"].data_ptr(), s["cal_z"].data_ptr(),
            s["res_x"].data_ptr(), s["res_z"].data_ptr(), nt, n, case["dt"], C.byref(w),
            torch.cuda.current_stream().cuda_stream))
        return dict(misfit=w.value, res_x=s["res_x"], res_z=s["res_z"])
    fd = s["fd"]
    if do == "models":
        descs, which = [], []
        for k, p in enumerate(s["parts"]):
            descs.append(dict(vp=p["m"]["vp0"], vs=p["m"]["vs0"], rho=p["m"]["rho0"], nt=p["nt"]))
            for d, (z, x) in zip(p["shots"], p["obs"]):
                _enqueue(case, fd, d, z.array, x.array, nt=p["nt"])
                which.append(k)
        per, grads = fd.run_models(descs, which)
        return dict(per=per, grads=[list(g[:3]) for g in grads])
    m, shots, obs = s["m"], s["shots"], s["obs"]
    if do == "turn":
        # the order of the reference driver's calls, shot by shot (main.cpp:585-631)
        misfit = 0.0
        pml = case["pml"]
        for d, (z, x) in zip(shots, obs):
            fd.ntr = d["ntr"]
            fd.isx, fd.isz, fd.igz = d["isx"], pml + 2, pml
            fd.ngx_left, fd.delta_left, fd.record_left_in_v = d["ngx_left"], d["delta_left"], 0
            fd.record_copytoGPU(z.array, x.array, d["gc"])
            fd.bufferVpVsHtoD(d["delta_left"])
            misfit = sg.IMAGE_SINGLESHOT(fd, misfit)
        return dict(misfit=misfit, grads=fd.imagebuffer_resettozero())
    if do == "hessian":
        for d in shots:
            _enqueue(case, fd, d)
        # the vectors of a conjugate-gradient solve are models, in the models' 32 bits
        return [h.astype(np.float32) for h in fd.hessian_vector(m["dvp"], m["dvs"])]
    for i, d in enumerate(shots):
        z, x = obs[i] if obs else (None, None)
        _enqueue(case, fd, d, z.array if obs else None, x.array if obs else None)
    if do == "forward":
        fd.run_forward()
        out = {}
        for i, d in enumerate(shots):
            r = fd.read_records(i, ntr=d["ntr"])
            keys = ("syn_z", "syn_x") if case["stage"] == 1 else ("syn_z", "syn_x", "syn2_z", "syn2_x")
            for k in keys:
                out.setdefault(k, []).append(r[k].ravel())
        return {k: np.concatenate(v) for k, v in out.items()}
    if do == "search":
        g = m["dvp"], m["dvs"]
        tot, per = fd.line_search_parabola(g[0], g[1], -0.15, -0.75)
        return dict(misfits=tot, per=per)
    misfit, per = fd.run()
    out = dict(misfit=misfit, per=per)
    if case.get("rho"):
        out["rho"] = fd.read_density_gradient_f64()
    out["grads"] = fd.imagebuffer_resettozero()
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# FP32 bytes per padded cell and time step with every field read once and
# written once per time step (a step's two half-steps share what they read):
#   forward: v(2), sigma(3) in and out, lam, mu, 1/rho; Born: the scattered
#   fields (5) in and out, bp, bs
#   backward: reconstruction and adjoint fields (10) in and out, lam, mu,
#   1/rho, the three accumulators in and out (+ the density kernel's)
# and floating-point operations of the stencils and updates.
_FWD = {1: (52, 150), 2: (100, 330)}
_BWD = (116, 360)
_BWD_RHO = 8


def work(case):
    do = case["do"]
    if do == "ot":
        n = case["traces"] * case["nt"]
        return dict(bytes=24.0 * n, flops=2 * 60.0 * n)
    pml, nt = case["pml"], case["nt"]
    if do == "models":
        geo = random.Random(case["nx"] * 977 + case["nz"])
        csteps = 0
        for k in range(case["models"]):
            mx, mz, mt = case["nx"], case["nz"], nt
            if k:
                mx, mz, mt = (max(40, int(v * geo.uniform(0.45, 1.0))) for v in (mx, mz, mt))
            csteps += max(1, case["shots"] // case["models"]) * (mx + 2 * pml) * (mz + 2 * pml) * mt
    else:
        shots = _shots(case, case["nx"], case["shots"], 3)
        csteps = sum(d["nx"] + 2 * pml for d in shots) * (case["nz"] + 2 * pml) * nt
    fb, ff = _FWD[case["stage"]]
    if do == "forward":
        return dict(bytes=float(fb * csteps), flops=float(ff * csteps))
    if do == "search":
        return dict(bytes=3.0 * fb * csteps, flops=3.0 * ff * csteps)
    if do == "hessian":
        # L m (Born forward), the background forward with its kept velocities,
        # and one adjoint step: fields (5) in and out, the kept vx, vz, 3
        # coefficients, two FP64 accumulators in and out
        return dict(bytes=float((fb + 52 + 8 + 40 + 8 + 12 + 32) * csteps), flops=float((ff + 150 + 300) * csteps))
    bb, bf = _BWD
    if case.get("snap"):
        # adjoint only (5 fields in and out, lam, mu, 1/rho), and at every k-th
        # step vx, vz written and read and the accumulators in and out
        es = 4 if case["fmt"] == "f32" else 2
        bb, bf = 52 + (4 * es + 24) / case["snap"], 200
    elif case.get("rho"):
        bb += _BWD_RHO
    return dict(bytes=float((fb + bb) * csteps), flops=float((ff + bf) * csteps))


# ---------------------------------------------------------------------------
# the same in 64 bits: the equations written with torch, a group of shots of
# one width at a time
# ---------------------------------------------------------------------------
_K = (1225.0 / 1024.0, -245.0 / 3072.0, 49.0 / 5120.0, -5.0 / 7168.0)
_H = 4


def _diff(f, axis, plus):
    """8th-order staggered difference on the interior [4, n-4)^2 of the last two axes."""
    X, Z = f.shape[-2:]

    def at(o):
        ox, oz = (o, 0) if axis == 0 else (0, o)
        return f[..., _H + ox:X - _H + ox, _H + oz:Z - _H + oz]
    r = 0
    for k, c in enumerate(_K, 1):
        r = r + c * (at(k) - at(1 - k) if plus else at(k - 1) - at(-k))
    return r


def _whole(f):
    return torch.nn.functional.pad(f, (_H, _H, _H, _H))


class _Group:
    """Shots of one window width: coefficients, geometry and the two half-steps."""

    def __init__(self, case, stage, vp, vs, rho, dvp, dvs, shots, nz, nt, models=None):
        dev = "cuda"
        self.stage, self.nt = stage, nt
        pml = self.pml = case["pml"]
        self.dt, self.dx = float(np.float32(case["dt"])), float(np.float32(case["dx"]))
        nx = shots[0]["nx"]
        self.nx, self.nz, self.shots = nx, nz, shots
        X, Z = nx + 2 * pml, nz + 2 * pml
        cx = torch.arange(X, device=dev).clamp(pml, X - pml - 1) - pml
        cz = torch.arange(Z, device=dev).clamp(pml, Z - pml - 1) - pml
        left = torch.tensor([d["delta_left"] for d in shots], device=dev)
        t = lambda a: torch.as_tensor(a, device=dev, dtype=torch.float64)  # noqa: E731

        def cut(a):  # a: [allnx, allnz], or one such model per shot
            a = a if torch.is_tensor(a) else t(a)
            if a.dim() == 2:
                return a[left[:, None, None] + cx[None, :, None], cz[None, None, :]]
            s = torch.arange(len(shots), device=dev)
            return a[s[:, None, None], left[:, None, None] + cx[None, :, None], cz[None, None, :]]
        self.cut = cut
        self.vp, self.vs = cut(vp), cut(vs)
        self.rho = torch.full_like(self.vp, 2000.0) if stage == 2 else cut(rho)
        self.lam = self.rho * (self.vp ** 2 - 2 * self.vs ** 2)
        self.mu = self.rho * self.vs ** 2
        l10 = float(np.log10(np.float32(1.0) / np.float32(0.001)).astype(np.float32))

        def profile(n):
            i = np.arange(n)
            r = np.where(i < pml, (pml - i) / pml, np.where(i > n - pml, (i - (n - pml)) / pml, 0.0))
            return t((r.astype(np.float32) ** np.float32(4.0)).astype(np.float32))
        base = l10 * 5.0 * self.vp / (2.0 * pml)
        inn = (slice(None), slice(_H, -_H), slice(_H, -_H))
        self.inn = inn
        hx, hz = (0.5 * self.dt * (base * p)[inn] for p in (profile(X)[None, :, None], profile(Z)[None, None, :]))
        self.d1, self.d2, self.d3, self.d4 = 1 - hx, 1 + hx, 1 - hz, 1 + hz
        self.c = self.dt / self.dx
        self.ib, self.l, self.u = (1.0 / self.rho)[inn], self.lam[inn], self.mu[inn]
        self.l2m = self.l + 2 * self.u
        if stage == 2 and dvp is not None:
            self.born(dvp, dvs)
        S = len(shots)
        self.isx = torch.tensor([d["isx"] for d in shots], device=dev)
        self.isz, self.igz = pml + 2, pml
        self.s = torch.arange(S, device=dev)
        sh, rec, inj = [], [], []
        last = {}
        n = 0
        for k, d in enumerate(shots):
            for g in d["gc"]:
                o = np.float32(int(g) - d["ngx_left"])
                ij = pml + int(o / np.float32(self.dx))
                sh.append(k)
                rec.append(pml + int(o / np.float32(int(self.dx))) if stage == 2 else ij)
                inj.append(ij)
                last[(k, ij)] = n
                n += 1
        self.sh, self.rec = torch.tensor(sh, device=dev), torch.tensor(rec, device=dev)
        keep = sorted(last.values())  # of several traces injected at one cell the last counts
        self.keep = torch.tensor(keep, device=dev)
        self.ksh, self.kin = self.sh[self.keep], torch.tensor(inj, device=dev)[self.keep]
        self.zero = lambda: torch.zeros(S, X, Z, device=dev, dtype=torch.float64)  # noqa: E731
        self.zin = lambda: torch.zeros(S, X - 2 * _H, Z - 2 * _H, device=dev, dtype=torch.float64)  # noqa: E731
        self.source = case.get("source")

    def born(self, dvp, dvs):
        self.bp = (2 * self.rho * self.vp * self.cut(dvp))[self.inn]
        self.bs = (2 * self.rho * self.vs * self.cut(dvs))[self.inn]

    def fields(self):
        # totals vx vz txx tzz txz; parts of each
        return [self.zero() for _ in range(5)], [self.zin() for _ in range(10)]

    def vel(self, f, q, sgn):
        cx = sgn * self.ib * self.c
        q[0] = (self.d1 * q[0] + cx * _diff(f[2], 0, True)) / self.d2
        q[1] = (self.d3 * q[1] + cx * _diff(f[4], 1, False)) / self.d4
        q[2] = (self.d1 * q[2] + cx * _diff(f[4], 0, False)) / self.d2
        q[3] = (self.d3 * q[3] + cx * _diff(f[3], 1, True)) / self.d4
        f[0], f[1] = _whole(q[0] + q[1]), _whole(q[2] + q[3])

    def grad(self, vx, vz):
        return _diff(vx, 0, False), _diff(vz, 1, False), _diff(vx, 1, True), _diff(vz, 0, True)

    def stress(self, f, q, sgn, born=None):
        a, b, c, d = self.grad(f[0], f[1])
        if born is not None:  # strains of the background
            A, B, Cc, D = (x * self.c for x in born)
            mix = self.bp - 2 * self.bs
            add = (self.bp * A, mix * B, mix * A, self.bp * B, self.bs * D, self.bs * Cc)
            for k in range(6):
                q[4 + k] = q[4 + k] + add[k]
        k = sgn * self.c
        q[4] = (self.d1 * q[4] + k * self.l2m * a) / self.d2
        q[5] = (self.d3 * q[5] + k * self.l * b) / self.d4
        q[6] = (self.d1 * q[6] + k * self.l * a) / self.d2
        q[7] = (self.d3 * q[7] + k * self.l2m * b) / self.d4
        q[8] = (self.d1 * q[8] + k * self.u * d) / self.d2
        q[9] = (self.d3 * q[9] + k * self.u * c) / self.d4
        f[2], f[3], f[4] = _whole(q[4] + q[5]), _whole(q[6] + q[7]), _whole(q[8] + q[9])
        return a, b, c, d

    def bands(self):
        p, X, Z = self.pml, self.nx + 2 * self.pml, self.nz + 2 * self.pml
        x, z = slice(p, X - p), slice(p, Z - p)
        return [(slice(None), x, slice(p - _H, p + _H)), (slice(None), x, slice(Z - p - _H, Z - p + _H)),
                (slice(None), slice(p - _H, p + _H), z), (slice(None), slice(X - p - _H, X - p + _H), z)]

    def forward(self, sou, born, keep=None, every=1):
        """Records [nrec][nt][traces]; keep "strips" or "snaps" for a backward pass."""
        F, Q = self.fields()
        G, R = self.fields() if born else (None, None)
        recs, kept = [], []
        for it in range(self.nt):
            if self.source != "vz":
                for k in (2, 3):
                    F[k] = F[k].clone()
                    F[k][self.s, self.isx, self.isz] += sou[it]
            self.vel(F, Q, 1)
            if self.source == "vz":
                F[1][self.s, self.isx, self.isz] += sou[it]
            st = self.stress(F, Q, 1)
            at = (self.sh, self.rec, self.igz)
            if born:
                self.vel(G, R, 1)
                self.stress(G, R, 1, st)
                recs.append(torch.stack([G[1][at], G[0][at], F[1][at], F[0][at]]))
            else:
                recs.append(torch.stack([F[1][at], F[0][at]]))
            if keep == "snaps" and it % every == 0:
                kept.append((F[0], F[1]))
            elif keep == "strips":
                kept.append([(F[0][b].clone(), F[1][b].clone()) for b in self.bands()])
        return torch.stack(recs, 1), F, Q, kept

    def backward(self, F, Q, kept, rz, rx, snap, want_rho):
        """Time sums of the Vp and Vs gradients, illumination (and density kernel) per window cell."""
        p, w = self.pml, 1
        sgn = 1 if self.stage == 1 else -1
        A = [self.zero() for _ in range(5)]
        B = [self.zin() for _ in range(8)]
        i = (slice(None), slice(p, p + self.nx), slice(p, p + self.nz))
        j = (slice(None), slice(p - _H, p - _H + self.nx), slice(p - _H, p - _H + self.nz))
        gl, gm, il, rh = (torch.zeros_like(self.vp[i]) for _ in range(4))
        l2m = self.lam + 2 * self.mu
        for it in range(self.nt - 1, -1, -1):
            image = True
            if snap:
                image = it % snap == 0
                if image:
                    vx, vz = kept[it // snap]
                    st, w = self.grad(vx, vz), snap
                    F = [vx, vz]
            else:
                before = F[0], F[1]
                F[0], F[1] = F[0].clone(), F[1].clone()
                for b, (bx, bz) in zip(self.bands(), kept[it]):
                    F[0][b], F[1][b] = bx, bz
                st = self.stress(F, Q, -1)
                self.vel(F, Q, -1)
            A[1][self.ksh, self.kin, self.igz] = rz[it, self.keep]
            A[0][self.ksh, self.kin, self.igz] = rx[it, self.keep]
            a, b, c, d = self.grad(A[0], A[1])
            k = sgn * self.c
            B[4] = (self.d1 * B[4] + k * a) / self.d2
            B[5] = (self.d3 * B[5] + k * b) / self.d4
            B[6] = (self.d1 * B[6] + k * d) / self.d2
            B[7] = (self.d3 * B[7] + k * c) / self.d4
            A[2], A[3], A[4] = _whole(B[4]), _whole(B[5]), _whole(B[6] + B[7])
            P, R, T = l2m * A[2] + self.lam * A[3], self.lam * A[2] + l2m * A[3], self.mu * A[4]
            cx = sgn * self.ib * self.c
            B[0] = (self.d1 * B[0] + cx * _diff(P, 0, True)) / self.d2
            B[1] = (self.d3 * B[1] + cx * _diff(T, 1, False)) / self.d4
            B[2] = (self.d1 * B[2] + cx * _diff(T, 0, False)) / self.d2
            B[3] = (self.d3 * B[3] + cx * _diff(R, 1, True)) / self.d4
            A[0], A[1] = _whole(B[0] + B[1]), _whole(B[2] + B[3])
            if not image:
                continue
            gxx, gzz, gxz, gzx = (x[j] / self.dx for x in st)
            xx, zz, xz = A[2][i], A[3][i], A[4][i]
            gl -= w * (gxx + gzz) * (xx + zz)
            gm -= w * (2 * (gxx * xx + gzz * zz) + (gxz + gzx) * xz)
            il += w * (F[0][i] ** 2 + F[1][i] ** 2)
            if want_rho:
                rh -= (A[0][i] * (before[0] - F[0])[i] + A[1][i] * (before[1] - F[1])[i]) / self.dt
        vp, vs, rho = self.vp[i], self.vs[i], self.rho[i]
        return 2 * vp * rho * gl, -4 * vs * rho * gl + 2 * vs * rho * gm, il, rh


def _ot64(kind, dt, cal, obs, scale):
    """W2 misfit and half its gradient, per trace of [traces, nt] in 64 bits."""
    n = cal.shape[1]
    sig = torch.where(scale > 0, scale, torch.ones_like(scale))[:, None]
    if kind == 2:
        p, q, dp = cal ** 2 + 1e-3 * sig ** 2, obs ** 2 + 1e-3 * sig ** 2, 2 * cal
    else:
        p = torch.exp((cal - cal.amax(1, True)) / sig)
        q = torch.exp((obs - obs.amax(1, True)) / sig)
        dp = p / sig
    S = p.sum(1, True)
    f, g = p / S, q / q.sum(1, True)
    F, G = f.cumsum(1), g.cumsum(1)
    m = torch.searchsorted(G, F, right=True).clamp(max=n - 1)
    gm = g.gather(1, m)
    below = torch.where(m > 0, G.gather(1, (m - 1).clamp(min=0)), torch.zeros_like(gm))
    k = torch.arange(1, n + 1, device=cal.device, dtype=torch.float64)
    r = dt * (k - m - (F - below) / gm)
    q2 = r * f * dt / gm
    A = r ** 2 - 2 * q2.flip(1).cumsum(1).flip(1)
    return (r ** 2 * f).sum(1), 0.5 * (A - (f * A).sum(1, True)) / S * dp


def _ot_scale(kind, obs, group):
    """max |obs| per trace, floored at 1e-3 of its gather's (or the gather's)."""
    s = obs.abs().amax(1)
    out = torch.empty_like(s)
    for a, b in group:
        top = s[a:b].max()
        out[a:b] = top if kind == 3 else torch.maximum(s[a:b], 1e-3 * top)
    return out


def _groups(shots):
    by = {}
    for i, d in enumerate(shots):
        by.setdefault(d["nx"], []).append(i)
    return list(by.values())


def _exact_grads(case, m, shots, obs, nx, nz, nt, stage, misfit):
    sou = torch.as_tensor(synth.ricker(nt, case["dt"], case["f0"]), device="cuda", dtype=torch.float64)
    out = [torch.zeros(nx, nz, device="cuda", dtype=torch.float64) for _ in range(4)]
    per = [0.0] * len(shots)
    kind = _KINDS[misfit]
    for idx in _groups(shots):
        sel = [shots[i] for i in idx]
        g = _Group(case, stage, m["vp0"], m["vs0"], m["rho0"], m["dvp"], m["dvs"], sel, nz, nt)
        recs, F, Q, kept = g.forward(sou, stage == 2, "snaps" if case.get("snap") else "strips", case.get("snap", 1))
        o = [torch.cat([torch.as_tensor(np.array(obs[i][c].array), device="cuda", dtype=torch.float64) for i in idx])
             for c in (0, 1)]  # [traces, nt]
        pred = [(recs[c] + recs[c + 2] if stage == 2 else recs[c]).T for c in (0, 1)]
        ends, n = [], 0
        for d in sel:
            ends.append((n, n + d["ntr"]))
            n += d["ntr"]
        if kind == 0:
            res = [a - b for a, b in zip(pred, o)]
            w = sum((r ** 2).sum(1) for r in res)
        else:
            w, res = 0, []
            for a, b in zip(pred, o):
                ww, r = _ot64(kind, g.dt, a, b, _ot_scale(kind, b, ends))
                w = w + ww
                res.append(r)
        for i, (a, b) in zip(idx, ends):
            per[i] = float(w[a:b].sum())
        gr = g.backward(F, Q, kept, res[0].T.contiguous(), res[1].T.contiguous(), case.get("snap"), case.get("rho"))
        for k, d in enumerate(sel):
            x0 = d["delta_left"]
            for dst, src in zip(out, gr):
                dst[x0:x0 + d["nx"]] += src[k]
        del F, Q, kept, gr
    return per, [x.cpu().numpy() for x in out]


def _seconds(case):
    """Roughly what exact() takes: torch launches of a step, and FP64 arrays through memory."""
    pml = case["pml"]
    shots = _shots(case, case["nx"], case["shots"], 3) if case["do"] != "models" else []
    groups = _groups(shots)
    cells = sum(d["nx"] + 2 * pml for d in shots) * (case["nz"] + 2 * pml)
    half = 1 if case["do"] in ("forward", "search") else 3
    born = 1.6 if case["stage"] == 2 else 1.0
    if case["do"] == "search":
        cells *= 3
    return half * born * case["nt"] * (0.9e-3 * len(groups) + 1.5e-9 * cells)


def exact(case, seed):
    do = case["do"]
    if do == "ot":
        s = _gathers(case, seed)
        w, out = 0.0, {}
        for c in ("x", "z"):
            obs, cal = s["obs_" + c].double(), s["cal_" + c].double()
            sc = _ot_scale(case["kind"], obs, [(0, len(obs))])
            for a in range(0, len(obs), 512):
                ww, r = _ot64(case["kind"], float(np.float32(case["dt"])), cal[a:a + 512], obs[a:a + 512], sc[a:a + 512])
                w += float(ww.sum())
                out.setdefault("res_" + c, []).append(r)
        return dict(misfit=w, **{k: torch.cat(v) for k, v in out.items()})
    if do == "models" or _seconds(case) > 15:
        return None
    s = _inputs(case, seed)
    m, shots, obs = s["m"], s["shots"], s["obs"]
    nx, nz, nt, stage = case["nx"], case["nz"], case["nt"], case["stage"]
    sou = torch.as_tensor(synth.ricker(nt, case["dt"], case["f0"]), device="cuda", dtype=torch.float64)
    if do == "hessian":
        # H m = L^T (L m): the gradient of |L m|^2 / 2 by reverse-mode differentiation
        X, Z = max(d["nx"] for d in shots) + 2 * case["pml"], nz + 2 * case["pml"]
        if len(_groups(shots)) > 1 or 90.0 * 8 * len(shots) * X * Z * nt > 120e9:
            return None
        g = _Group(case, 2, m["vp0"], m["vs0"], None, None, None, shots, nz, nt)
        v = [torch.as_tensor(m[k], device="cuda", dtype=torch.float64).requires_grad_(True) for k in ("dvp", "dvs")]
        g.born(*v)
        recs = g.forward(sou, True)[0]
        (0.5 * (recs[:2] ** 2).sum()).backward()
        return [x.grad for x in v]
    with torch.no_grad():
        if do == "forward":
            out = {}
            parts = [None] * len(shots)
            for idx in _groups(shots):
                key = ("vp", "vs", "rho") if stage == 1 else ("vp0", "vs0", "rho0")
                g = _Group(case, stage, *(m[k] for k in key), m["dvp"], m["dvs"], [shots[i] for i in idx], nz, nt)
                recs = g.forward(sou, stage == 2)[0]
                a = 0
                for i in idx:
                    parts[i] = recs[:, :, a:a + shots[i]["ntr"]]
                    a += shots[i]["ntr"]
            for c, k in enumerate(("syn_z", "syn_x", "syn2_z", "syn2_x")[:4 if stage == 2 else 2]):
                out[k] = torch.cat([p[c].T.reshape(-1) for p in parts])
            return out
        if do == "search":
            per = np.zeros((len(shots), 3))
            for k, step in enumerate((0.0, -0.15, -0.75)):
                f = lambda a, b: a.astype(np.float64) - float(np.float32(step)) * b  # noqa: E731
                vp, vs = f(m["vp0"], m["dvp"]), f(m["vs0"], m["dvs"])
                for idx in _groups(shots):
                    g = _Group(case, 1, vp, vs, m["rho0"], None, None, [shots[i] for i in idx], nz, nt)
                    recs, a = g.forward(sou, False)[0], 0
                    for i in idx:
                        r = recs[:, :, a:a + shots[i]["ntr"]]
                        a += shots[i]["ntr"]
                        per[i, k] = sum(float(((r[c].T - torch.as_tensor(np.array(obs[i][c].array), device="cuda")
                                                .double()) ** 2).sum()) for c in (0, 1))
            return dict(misfits=per.sum(0), per=per)
        per, gr = _exact_grads(case, m, shots, obs, nx, nz, nt, stage, case["misfit"])
    if do == "turn":
        return dict(misfit=sum(per), grads=tuple(gr[:3]))
    out = dict(misfit=sum(per), per=np.array(per), grads=tuple(gr[:3]))
    if case.get("rho"):
        out["rho"] = gr[3]
    return out
