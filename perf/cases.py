"""Workloads of the stepper as its users run it, through the package's public
entry points, for timing and for comparing two builds.

Four ways of use, each a `kind`:
  shot    one whole job: Simulation(config, medium), run(nt), the five
          seismograms (and the snapshots the configuration asks for), close
  window  a resident simulation advanced by one window of steps, whose
          seismogram window is streamed to page-locked host memory
  batch   several shots as one Batch: create, run(nt), seismograms, close
  server  a list of requests submitted to a running Server, waited for and read

Media: "layered" and "uniform" (few distinct materials), "borehole" (the
reference program's model), "lognormal" (every cell different).
"""
import ctypes
import math

import numpy as np
import torch

from mixedprecisionfaracoustic_b200 import Batch, Medium, Server, ShotConfig, Simulation
from mixedprecisionfaracoustic_b200 import biot, presets
from mixedprecisionfaracoustic_b200._abi import SRC_P, SRC_TAU

COMPONENTS = ("txx", "tzz", "vux", "vwx", "p")
DX, DT = presets.DX, presets.DT
BATCH_SIZES = ((1024, 1024), (1536, 1024), (2048, 2048), (3072, 1536))


def _case(name, kind, dim, n, order, precision, medium, steps, nrec, rounding="fast", npml=20, nshots=1, warm=0):
    c = {"name": name} if name else {}
    return c | {"kind": kind, "dim": dim, "nx": n[0], "ny": n[1] if dim == 3 else 1, "nz": n[-1],
                "npml": npml, "order": order, "precision": precision, "rounding": rounding, "medium": medium,
                "steps": steps, "warm": warm, "nrec": nrec, "nshots": nshots}


def listed():
    return [
        # a quick look at a small section: step latency, launches and set-up
        _case("shot2d_small_fp32", "shot", 2, (256, 192), 2, "fp32", "layered", 500, 64),
        # a mid-size 2D request with ragged extents, alone on the device
        _case("shot2d_ragged_fp32", "shot", 2, (777, 1033), 2, "fp32", "layered", 1000, 256),
        # the 2D layered benchmark model as one job
        _case("shot2d_large_fp32", "shot", 2, (4000, 2000), 2, "fp32", "layered", 2000, 2000),
        # the same model in the reference's compensated half storage, mid-run
        _case("window2d_large_comp16", "window", 2, (4000, 2000), 2, "comp16", "layered", 100, 500, warm=150),
        # a heterogeneous section, odd extents, fourth order, bf16 storage
        _case("window2d_het_cbf16_o4", "window", 2, (3001, 1507), 4, "cbf16", "lognormal", 100, 500, warm=150),
        # the accuracy reference users check the reduced precisions against
        _case("shot2d_fp64", "shot", 2, (1000, 500), 2, "fp64", "layered", 500, 256),
        # the 3D homogeneous model, fourth order, mid-run
        _case("window3d_fp32_o4", "window", 3, (160, 160, 160), 4, "fp32", "uniform", 50, 128, warm=100),
        # 3D heterogeneous in compensated half storage
        _case("window3d_het_comp16", "window", 3, (256, 256, 192), 2, "comp16", "lognormal", 20, 128, warm=100),
        # the large 3D heterogeneous model (the biggest state here)
        _case("window3d_het_fp32", "window", 3, (384, 384, 288), 2, "fp32", "lognormal", 10, 128, warm=100),
        # the reference program's own run (borehole, its rounding, its snapshot)
        _case("shot3d_reference_fp32", "shot", 3, (128, 128, 128), 2, "fp32", "borehole", 600, 192,
              rounding="reference", npml=32),
        # a survey's shots together: sizes of the batched configuration
        _case("batch2d_fp32", "batch", 2, (3072, 2048), 2, "fp32", "layered", 500, 256, nshots=8),
        # serving: 2D and 3D requests of different sizes and lengths at once
        _case("server_mixed_fp32", "server", 2, (1200, 1200), 2, "fp32", "layered", 400, 64, nshots=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("shot", "window", "batch", "server"), (0.35, 0.4, 0.13, 0.12))[0]
    order = rng.choice((2, 2, 4))
    if kind == "shot":
        dim = rng.choice((2, 2, 3))
        precision = rng.choices(("fp32", "comp16", "cbf16", "fp64"), (0.5, 0.25, 0.15, 0.1))[0]
        rounding = "reference" if precision == "fp32" and rng.random() < 0.25 else "fast"
        if dim == 2:
            n = (_log_int(rng, 200, 2600), 1, _log_int(rng, 150, 1800))
            steps = rng.randint(300, 1000)
            return _case(None, kind, 2, (n[0], n[2]), order, precision, rng.choice(("layered", "layered", "lognormal")),
                         steps, _log_int(rng, 16, min(512, n[0])), rounding)
        n = tuple(_log_int(rng, 40, 176) for _ in range(3))
        return _case(None, kind, 3, n, order, precision, rng.choice(("uniform", "borehole", "lognormal")),
                     rng.randint(150, 300), _log_int(rng, 8, min(128, n[0])), rounding)
    if kind == "window":
        precision = rng.choices(("fp32", "comp16", "cbf16", "fp64"), (0.4, 0.3, 0.2, 0.1))[0]
        if rng.random() < 0.5:
            n = (_log_int(rng, 1200, 4000), 1, _log_int(rng, 900, 2000))
            return _case(None, kind, 2, (n[0], n[2]), order, precision, rng.choice(("layered", "lognormal")),
                         rng.randint(40, 100), 256, warm=120)
        n = tuple(_log_int(rng, 96, 288) for _ in range(3))
        return _case(None, kind, 3, n, order, precision, rng.choice(("uniform", "lognormal")), rng.randint(10, 25), 96,
                     warm=80)
    precision = rng.choice(("fp32", "fp32", "comp16", "cbf16"))
    if kind == "batch":
        n = (_log_int(rng, 600, 2600), _log_int(rng, 500, 1800))
        return _case(None, kind, 2, n, order, precision, "layered", rng.randint(300, 500), 128,
                     nshots=rng.randint(2, 8))
    n = (_log_int(rng, 512, 1400), _log_int(rng, 512, 1400))
    return _case(None, kind, 2, n, 2, precision, "layered", rng.randint(200, 400), 64,
                 nshots=rng.randint(3, 8))


# ---------------------------------------------------------------------------
# inputs


def _smooth(shape, gen, dev, corr=10):
    """A unit-variance smooth field: coarse white noise, linearly interpolated."""
    coarse = [s // corr + 2 for s in shape]
    g = torch.randn([1, 1] + coarse, generator=gen, device=dev)
    mode = "bilinear" if len(shape) == 2 else "trilinear"
    g = torch.nn.functional.interpolate(g, size=list(shape), mode=mode, align_corners=True)[0, 0]
    return (g - g.mean()) / g.std()


def _lognormal(shape, seed):
    """Log-normal perturbation (sigma 0.1) of the homogeneous model's moduli and
    permeability, as host arrays, with the fast P velocity bound."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    gen = torch.Generator(device=dev).manual_seed(seed)
    p = presets.C0
    f = [torch.exp(0.1 * _smooth(shape, gen, dev) - 0.005) for _ in range(4)]
    ks, kb = p["Ks"] * f[0], p["Kb"] * f[1]
    kb = torch.minimum(kb, 0.95 * ks)
    mu = p["mu"] * f[2]
    phi, kf, rhof = p["phi"], p["Kf"], p["rhof"]
    alpha = 1 - kb / ks
    m = kf * ks / (phi * ks + (alpha - phi) * kf)
    h = alpha * alpha * m + kb + mu * (4.0 / 3.0)
    rho = (1 - phi) * p["rhos"] + phi * rhof
    full = lambda v: np.full(shape, v, dtype=np.float32)   # noqa: E731
    host = lambda t: t.float().contiguous().cpu().numpy()  # noqa: E731
    vmax = math.sqrt(float(h.max()) / rho) * 1.05
    med = Medium({"rho": full(rho), "rhof": full(rhof), "M": host(m), "C": host(alpha * m), "H": host(h),
                  "H2mu": host(h - 2 * mu), "mu": host(mu), "C1": host(p["eta"] / (p["kappa"] * f[3])),
                  "C2": full((1 + 2 / p["m_shape"]) * p["tort"] * rhof / phi)})
    return med, vmax


def _medium(c, nx, ny, nz, seed):
    shape = (nz, ny, nx) if c["dim"] == 3 else (nz, nx)
    if c["medium"] == "lognormal":
        return _lognormal(shape, seed)
    if c["medium"] == "layered":
        return presets.layered_medium(nx, nz, seed, depth_scale=nz / 2000.0)
    scale = 1.0 + 0.05 * (np.random.RandomState(seed % (1 << 31)).random_sample() - 0.5)
    if c["medium"] == "borehole":
        med = biot.reference_borehole_medium(nx, ny, nz)
        for k in ("M", "C", "H", "H2mu", "mu"):
            med[k] = med[k] * np.float32(scale)
        return med, 4000.0
    p = dict(presets.C0)
    p["Kb"] *= scale
    p["mu"] *= scale
    co = biot.biot_from_moduli(p["Ks"], p["Kb"], p["mu"], p["Kf"], p["rhos"], p["rhof"], p["phi"], p["tort"],
                               p["eta"], p["kappa"], p["m_shape"])
    return presets.uniform_medium(shape, co), math.sqrt(co["H"] / co["rho"]) * 1.05


def _one(c, seed, dim=None, n=None, steps=None, nt=None, medium=None):
    """(ShotConfig, Medium) of one shot of the case."""
    c = dict(c, dim=dim or c["dim"], medium=medium or c["medium"])
    nx, ny, nz = n or (c["nx"], c["ny"], c["nz"])
    npml, steps = c["npml"], steps or c["steps"]
    med, vmax = _medium(c, nx, ny, nz, seed)
    r = np.random.RandomState((seed * 7 + 3) % (1 << 31))
    nrec = min(c["nrec"], nx)
    rx = [npml + (i * nx) // nrec for i in range(nrec)]
    cy = npml + ny // 2 if c["dim"] == 3 else 0
    if c["medium"] == "borehole":     # the reference program's geometry and units
        sx, sz = npml + nx // 2, npml + min(20, nz // 2)
        nzp = nz + 2 * npml
        return ShotConfig(dim=3, nx=nx, ny=ny, nz=nz, npml=npml, order=c["order"], precision=c["precision"],
                          nt=nt or steps, dx=0.01, dt=0.9e-6, f0=3000.0, t0=1.2 / 3000.0, pml_v0=vmax, pml_r=1e-6,
                          src=(sx, cy, sz), src_mask=SRC_TAU, rec_x=[sx] * (nzp - 4), rec_y=[cy] * (nzp - 4),
                          rec_z=list(range(2, nzp - 2)), snap_steps=[steps - 1], snap_fields=["txx"], snap_y=cy,
                          rounding=c["rounding"]), med
    f0 = 30.0 + 10.0 * r.random_sample()
    sx = npml + nx // 4 + int(r.randint(0, max(1, nx // 2)))
    sz = npml + (nz // 2 if c["dim"] == 3 else min(10, nz - 1))
    return ShotConfig(dim=c["dim"], nx=nx, ny=ny, nz=nz, npml=npml, order=c["order"], precision=c["precision"],
                      nt=nt or steps, dx=DX, dt=DT, f0=f0, pml_v0=vmax, pml_r=1e-6, src=(sx, cy, sz),
                      src_mask=SRC_TAU | SRC_P, rec_x=rx, rec_y=[cy] * nrec, rec_z=[sz] * nrec, check_cfl=1,
                      rounding=c["rounding"]), med


def _parts(c):
    """The shots of a batch or server case: (dim, (nx, ny, nz), steps) each."""
    if c["kind"] == "batch":
        return [(2, (max(64, c["nx"] * BATCH_SIZES[i % 4][0] // 3072), 1, max(64, c["nz"] * BATCH_SIZES[i % 4][1] // 2048)),
                 c["steps"]) for i in range(c["nshots"])]
    out = []
    for i in range(c["nshots"]):
        if i % 3 == 2:                                 # every third request is 3D
            e = max(48, min(128, (c["nx"] + 37 * i) // 12))
            out.append((3, (e, e, e), max(50, c["steps"] // 2)))
        else:
            out.append((2, (int(c["nx"] * (1 - 0.07 * i)), 1, int(c["nz"] * (1 - 0.05 * (i % 5)))), c["steps"] - 17 * i))
    return out


def _jobs(c, seed):
    if c["kind"] in ("shot", "window"):
        return [_one(c, seed, nt=_window_nt(c) if c["kind"] == "window" else None)]
    return [_one(c, seed * 31 + i, dim=d, n=n, steps=s, medium="uniform" if d == 3 else c["medium"])
            for i, (d, n, s) in enumerate(_parts(c))]


def _padded(c, n=None, dim=None):
    nx, ny, nz = n or (c["nx"], c["ny"], c["nz"])
    p = 2 * c["npml"]
    return (nx + p, ny + p if (dim or c["dim"]) == 3 else 1, nz + p)


def _window_nt(c):
    """Length of a streamed recording: long enough for some seconds of windows."""
    return int(max(4000, 2e11 / np.prod(_padded(c), dtype=float)))


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=torch.cuda.is_available())


def prepare(case, seed):
    jobs = _jobs(case, seed)
    st = {"case": case, "jobs": jobs}
    if case["kind"] == "window":
        cfg, med = jobs[0]
        st["sim"] = Simulation(cfg, med)
        st["sim"].run(case["warm"])
        st["sim"].sync()
        st["jobs"] = [(cfg, None)]                     # the host medium is no longer needed
        st["out"] = [_pinned((cfg.nrec, case["steps"])) for _ in COMPONENTS]
    elif case["kind"] == "shot":
        cfg = jobs[0][0]
        st["out"] = [_pinned((cfg.nrec, cfg.nt)) for _ in COMPONENTS]
    elif case["kind"] == "server":
        st["server"] = Server(16 << 30)
    return st


# ---------------------------------------------------------------------------
# one pass


def run(state):
    kind = state["case"]["kind"]
    if kind == "window":
        sim, k = state["sim"], state["case"]["steps"]
        it = sim.step
        sim.run(k)
        for comp, o in zip(COMPONENTS, state["out"]):
            sim.copy_traces_async(comp, it, o.numpy())
        sim.sync()
        return state["out"]
    if kind == "shot":
        cfg, med = state["jobs"][0]
        with Simulation(cfg, med) as sim:
            sim.run(cfg.nt)
            for comp, o in zip(COMPONENTS, state["out"]):
                sim.traces(comp, o.numpy())
            snaps = [sim.snapshot(k, f) for k in range(len(cfg.snap_steps)) for f in cfg.snap_fields]
        return list(state["out"]) + snaps
    if kind == "batch":
        cfgs = [j[0] for j in state["jobs"]]
        b = Batch(cfgs, [j[1] for j in state["jobs"]])
        b.run(max(c.nt for c in cfgs))
        b.sync()
        out = [np.stack([b.traces(i, comp) for comp in COMPONENTS]) for i in range(len(cfgs))]
        b.close()
        return out
    srv = state["server"]
    ids = [srv.submit(cfg, med) for cfg, med in state["jobs"]]
    out = []
    for rid in ids:
        srv.wait(rid)
        out.append(np.stack([srv.traces(rid, comp) for comp in COMPONENTS]))
        srv.release(rid)
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _step_work(c, dim, n):
    """(bytes, flops) of one time step of one shot: each state value read once
    and written once, the medium read once (one byte a cell where few distinct
    materials exist, else the nine input arrays)."""
    e = _padded(c, n, dim)
    cells = float(np.prod(e, dtype=float))
    value = {"fp32": 4, "fp64": 8, "comp16": 3, "cbf16": 3}[c["precision"]]
    fields, slots = (13, 4) if dim == 3 else (8, 3)
    medium = 36 if c["medium"] == "lognormal" else 1
    b = cells * (fields * 2 * value + medium)
    real = 8 if c["precision"] == "fp64" else 4
    for ax in (range(3) if dim == 3 else (0, 2)):      # absorbing slabs: two memory variables a difference
        b += cells / e[ax] * 2 * c["npml"] * 2 * slots * 2 * 2 * real
    return b, cells * (150 if dim == 3 else 70) * (1.6 if c["order"] == 4 else 1.0)


def work(case):
    c = case
    if c["kind"] in ("shot", "window"):
        parts = [(c["dim"], (c["nx"], c["ny"], c["nz"]), c["steps"])]
    else:
        parts = _parts(c)
    total = [0.0, 0.0]
    for dim, n, steps in parts:
        b, f = _step_work(dict(c, medium="uniform" if c["kind"] == "server" else c["medium"]), dim, n)
        total[0] += b * steps + steps * 5 * 4 * min(c["nrec"], n[0])
        total[1] += f * steps
        if c["kind"] != "window":                      # the medium comes from the host once
            total[0] += 36.0 * n[0] * n[1] * n[2]
    return {"bytes": total[0], "flops": total[1]}


# ---------------------------------------------------------------------------
# the same answers in 64 bits with plain torch


def _f32(v):
    """A configuration value as the C ABI holds it."""
    return float(ctypes.c_float(v).value)


def _absorb(n, np_, h, dt, v0, rc):
    """(b, e, b_half, e_half, first interior cell, first right cell) of one axis."""
    h32 = np.float32(h)
    dp = np.float32(np_) * h32
    right = np.float32(n - 1) * h32 - dp
    i = np.arange(n)
    x32 = i.astype(np.float32) * h32
    inl = (x32 >= 0) & (x32 < dp)
    inr = (x32 >= right) & (x32 < np.float32(n) * h32)
    if np_ == 0:
        inl[:] = inr[:] = False
    x = i * float(h32)
    d0 = 3.0 * v0 * math.log(1.0 / rc) / (2.0 * float(dp)) if np_ else 0.0
    d, dh = np.zeros(n), np.zeros(n)
    if np_:
        d[inl] = d0 * ((float(dp) - x[inl]) / float(dp)) ** 2
        dh[inl] = d0 * ((float(dp) - x[inl] - 0.5 * h) / float(dp)) ** 2
        d[inr] = d0 * ((x[inr] - float(right)) / float(dp)) ** 2
        dh[inr] = d0 * ((x[inr] + 0.5 * h - float(right)) / float(dp)) ** 2
    lo = int(np.max(np.nonzero(inl)[0]) + 1) if inl.any() else 0
    hi = int(np.min(np.nonzero(inr)[0])) if inr.any() else n
    return -dt * d * 0.5, np.exp(-d * dt), -dt * dh * 0.5, np.exp(-dh * dt), lo, hi


class _Plain:
    """The scheme in double precision: staggered differences of order 2 or 4,
    CPML memory variables on the slabs, one shot."""

    def __init__(self, cfg, med, dev):
        self.cfg, self.dev, self.dim = cfg, dev, cfg.dim
        self.hw = cfg.order // 2
        ex = cfg.padded
        self.shape = (ex[2], ex[1], ex[0]) if cfg.dim == 3 else (ex[2], ex[0])
        self.axes = {"z": 0, "y": 1, "x": 2} if cfg.dim == 3 else {"z": 0, "x": 1}
        self.h, self.dt = _f32(cfg.dx), _f32(cfg.dt)
        self._coefficients(med)
        self.f = {}
        for k in ("vux", "vuz", "vwx", "vwz", "p", "txx", "tzz", "txz") + (
                ("vuy", "vwy", "tyy", "txy", "tyz") if cfg.dim == 3 else ()):
            self.f[k] = torch.zeros(self.shape, dtype=torch.float64, device=dev)
        self.abs, self.mem = {}, {}
        for name, ax in self.axes.items():
            b, e, bh, eh, lo, hi = _absorb(self.shape[ax], cfg.npml, self.h, self.dt, _f32(cfg.pml_v0), _f32(cfg.pml_r))
            hw, n = self.hw, self.shape[ax]
            view = [1] * len(self.shape)
            view[ax] = -1
            sides = []
            for a0, a1 in ((hw, min(lo, n - hw)), (max(hi, hw), n - hw)):
                if a1 > a0:
                    t = lambda v: torch.from_numpy(v[a0:a1].copy()).to(dev).view(view)  # noqa: E731
                    sides.append((a0 - hw, a1 - a0, (t(b), t(e)), (t(bh), t(eh))))
            self.abs[name] = sides

    def _pad(self, a):
        np_ = self.cfg.npml
        t = torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(self.dev)
        phys = (self.cfg.nz, self.cfg.ny, self.cfg.nx) if self.dim == 3 else (self.cfg.nz, self.cfg.nx)
        t = t.reshape(phys)
        for ax, n in enumerate(phys):
            t = t.index_select(ax, (torch.arange(n + 2 * np_, device=self.dev) - np_).clamp(0, n - 1))
        return t.double()

    def _in(self, t, **shift):
        """The updated cells of t, displaced along the named axes."""
        for name, ax in self.axes.items():
            t = t.narrow(ax, self.hw + shift.get(name, 0), self.shape[ax] - 2 * self.hw)
        return t

    def _coefficients(self, med):
        dt = self.dt
        self.c = {k: self._in(self._pad(med[k])).clone() for k in ("C", "M", "H", "H2mu", "rhof")}
        rho, c1, c2, mu = (self._pad(med[k]) for k in ("rho", "C1", "C2", "mu"))
        self.v = {}
        for a in self.axes:
            r = 2.0 / (self._in(rho) + self._in(rho, **{a: 1}))
            f1 = 0.5 * (self._in(c1) + self._in(c1, **{a: 1}))
            f2 = 0.5 * (self._in(c2) + self._in(c2, **{a: 1}))
            base = f2 - self.c["rhof"] ** 2 * r
            den = 0.5 * f1 * dt + base
            keep = f1 != 0
            inv = torch.where(keep, 1.0 / den, torch.zeros_like(den))
            self.v[a] = (r, (base - 0.5 * f1 * dt) * inv, dt * inv)
        self.mu = {}
        for a, b in (("x", "z"),) + ((("x", "y"), ("y", "z")) if self.dim == 3 else ()):
            q = [self._in(mu), self._in(mu, **{a: 1}), self._in(mu, **{b: 1}), self._in(mu, **{a: 1, b: 1})]
            none = (q[0] == 0) | (q[1] == 0) | (q[2] == 0) | (q[3] == 0)
            m = 4.0 / sum(1.0 / v for v in q)
            self.mu[a + b] = torch.where(none, torch.zeros_like(m), m) * dt

    def _d(self, field, a, fwd):
        """CPML-corrected staggered difference of a field along axis a at the updated cells."""
        t, o = self.f[field], (0 if fwd else -1)
        d = self._in(t, **{a: o + 1}) - self._in(t, **{a: o})
        if self.hw == 2:
            far = self._in(t, **{a: o + 2}) - self._in(t, **{a: o - 1})
            d.mul_(1.125 / self.h).add_(far, alpha=-1.0 / 24.0 / self.h)
        else:
            d.div_(self.h)
        ax = self.axes[a]
        for i, (start, length, whole, half) in enumerate(self.abs[a]):
            b, e = half if fwd else whole
            w = d.narrow(ax, start, length)
            key = (field, a, fwd, i)
            if key not in self.mem:
                self.mem[key] = (torch.zeros_like(w), torch.zeros_like(w))
            psi, prev = self.mem[key]
            prev.mul_(e).add_(w).mul_(b)
            psi.mul_(e).add_(prev)
            prev.copy_(w)
            w.add_(psi)
        return d

    def _velocity(self, a, total, dp):
        r, keep, dti = self.v[a]
        rr = self.c["rhof"] * r
        u, w = self._in(self.f["vu" + a]), self._in(self.f["vw" + a])
        new = w * keep - dti * (rr * total + dp)
        u.add_(r * total, alpha=self.dt).sub_(rr * (new - w))
        w.copy_(new)

    def step(self, sample):
        f, d = self.f, self._d
        c = self.cfg
        at = (c.src[2], c.src[1], c.src[0]) if self.dim == 3 else (c.src[2], c.src[0])
        if c.src_mask & SRC_TAU:
            for k in ("txx", "tyy", "tzz"):
                if k in f:
                    f[k][at] += sample
        if c.src_mask & SRC_P:
            f["p"][at] -= sample
        three = self.dim == 3
        total = {"x": d("txx", "x", True) + d("txz", "z", False)}
        total["z"] = d("tzz", "z", True) + d("txz", "x", False)
        if three:
            total["x"] += d("txy", "y", False)
            total["z"] += d("tyz", "y", False)
            total["y"] = d("tyy", "y", True) + d("txy", "x", False) + d("tyz", "z", False)
        for a in self.axes:
            self._velocity(a, total[a], d("p", a, True))
        del total
        e = {a: d("vu" + a, a, False) for a in self.axes}
        div, wdiv = sum(e.values()), sum(d("vw" + a, a, False) for a in self.axes)
        k, dt = self.c, self.dt
        self._in(f["p"]).sub_(k["C"] * div + k["M"] * wdiv, alpha=dt)
        base = k["H2mu"] * div + k["C"] * wdiv
        shear2 = k["H"] - k["H2mu"]
        for a in self.axes:
            if "t" + a + a in f:
                self._in(f["t" + a + a]).add_(base + shear2 * e[a], alpha=dt)
        for ab, m in self.mu.items():
            a, b = ab
            self._in(f["t" + ab]).add_(m * (d("vu" + a, b, True) + d("vu" + b, a, True)))


def _plain(cfg, med, first, steps):
    """Traces [5][nrec, steps] from step `first` on, and the final fields."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    s = _Plain(cfg, med, dev)
    f0 = _f32(cfg.f0)
    t0 = _f32(cfg.t0) if cfg.t0 > 0 else 1.2 / f0
    pi = 3.1415926535
    rx, ry, rz = (torch.tensor(list(v), device=dev) for v in (cfg.rec_x, cfg.rec_y, cfg.rec_z))
    at = (rz, ry, rx) if cfg.dim == 3 else (rz, rx)
    out = torch.zeros((5, cfg.nrec, steps), dtype=torch.float64, device=dev)
    for it in range(first + steps):
        a = it * s.dt - t0
        s.step(-(1 - 2 * pi * pi * f0 * f0 * a * a) * math.exp(-pi * pi * f0 * f0 * a * a))
        if it >= first:
            for q, comp in enumerate(COMPONENTS):
                out[q, :, it - first] = s.f[comp][at]
    return out, s.f


def exact(case, seed):
    c = case
    if c["kind"] in ("shot", "window"):
        cost = (c["steps"] + c["warm"]) * np.prod(_padded(c), dtype=float) * (2 if c["dim"] == 3 else 1)
    else:
        cost = sum(s * np.prod(_padded(c, n, d), dtype=float) * (2 if d == 3 else 1) for d, n, s in _parts(c))
    if cost > 5e10:
        return None
    if c["kind"] in ("batch", "server"):
        return [_plain(cfg, med, 0, cfg.nt)[0] for cfg, med in _jobs(c, seed)]
    cfg, med = _jobs(c, seed)[0]
    tr, fields = _plain(cfg, med, c["warm"], c["steps"])
    out = [tr[q] for q in range(5)]
    if c["kind"] == "shot" and len(cfg.snap_steps):
        out += [fields[f][:, cfg.snap_y, :].contiguous() for f in cfg.snap_fields]
    return out
