"""The work that users of this library have it do, for timing and comparing builds of it.

Every case goes through the public classes of rockseis_b200.rockseis.  `exact`
restates each path in float64 with plain torch (derivatives as banded matrices, the
whole forward history kept), without this library's code.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from rockseis_b200 import abi
from rockseis_b200 import rockseis as rs

PREC = {"exact": abi.F32_EXACT, "fast": abi.F32_FAST}
CKPT = {"native": abi.CKPT_NATIVE, "f16": abi.CKPT_F16, "bf16": abi.CKPT_BF16}
VMAX = 3600.0

# do: "call" the one-call modelling driver on host arrays (a batch where shots > 1),
# "plan" a batch kept on the device, "fwi" a resident gradient batch, "rtm" the
# one-call image driver.  ny = 0 in 2D.
BASE = dict(ny=0, dx=10.0, order=8, fs=False, shots=1, ncheck=0, ckpt="native", nhx=1)


def listed():
    def c(name, **kw):
        return dict(BASE, name=name, **kw)

    return [
        # a first trial shot on a toy grid with the classes' default arithmetic: launches and host work
        c("a2_toy_exact", do="call", phys="a2", prec="exact", nx=61, nz=41, lpml=12, nt=150, nrec=20),
        # one marine shot, the usual size of a 2D acoustic model: the state stays in L2
        c("a2_shot_fast", do="call", phys="a2", prec="fast", nx=501, nz=301, lpml=20, nt=2000, nrec=251),
        # a line of shots in uneven aperture windows under a free surface, default order and arithmetic
        c("a2_line_exact", do="call", phys="a2", prec="exact", nx=601, nz=201, lpml=20, nt=400, nrec=151, order=4,
          fs=True, shots=24),
        # the gradient an inversion computes at each iteration: shots resident, 16-bit checkpoints
        c("a2_fwi_fast", do="fwi", phys="a2", prec="fast", nx=601, nz=201, lpml=20, nt=700, nrec=301, shots=16,
          ncheck=40, ckpt="f16"),
        # one shot of a migration with extended lags, lossless checkpoints, odd sizes
        c("a2_rtm_exact", do="rtm", phys="a2", prec="exact", nx=353, nz=187, lpml=20, nt=600, nrec=177, nhx=5),
        # the elastic forward batch of the benchmark, fewer steps
        c("e2_plan_fast", do="plan", phys="e2", prec="fast", nx=801, nz=401, dx=5.0, lpml=30, nt=600, nrec=400,
          shots=16),
        # a few elastic shots bit for bit as the CPU code computes them, free surface
        c("e2_call_exact", do="call", phys="e2", prec="exact", nx=401, nz=301, dx=5.0, lpml=30, nt=400, nrec=150,
          fs=True, shots=4),
        # elastic gradient of a small batch
        c("e2_fwi_fast", do="fwi", phys="e2", prec="fast", nx=401, nz=251, lpml=20, nt=400, nrec=150, shots=4,
          ncheck=30, ckpt="f16"),
        # one 3D acoustic window in the default arithmetic
        c("a3_call_exact", do="call", phys="a3", prec="exact", nx=121, ny=111, nz=101, lpml=15, nt=80, nrec=100),
        # 3D acoustic shots in windows of varying size, resident
        c("a3_plan_fast", do="plan", phys="a3", prec="fast", nx=221, ny=201, nz=181, dx=12.5, lpml=20, nt=60, nrec=225,
          shots=4),
        # 3D elastic shots, resident
        c("e3_plan_fast", do="plan", phys="e3", prec="fast", nx=181, ny=161, nz=151, lpml=20, nt=60, nrec=100, shots=2),
        # 3D elastic gradient with BF16 checkpoints and few snapshots
        c("e3_fwi_fast", do="fwi", phys="e3", prec="fast", nx=121, ny=111, nz=101, lpml=20, nt=60, nrec=100, ncheck=10,
          ckpt="bf16"),
    ]


def draw(rng):
    """One more case: any of the listed kinds of work, its sizes spread over their range."""
    c = dict(rng.choice(listed()))
    c.pop("name")

    def size(hi, lo):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if c["ny"]:
        n = {"call": 150, "plan": 200, "fwi": 120}[c["do"]]
        c["nx"], c["ny"], c["nz"] = (size(n, 40) for _ in range(3))
        c["nt"] = size(80, 60)
        c["shots"] = rng.randint(1, 2) if c["do"] == "fwi" else rng.randint(1, {"a3": 4, "e3": 2}[c["phys"]])
    else:
        nxm, nzm = (801, 401) if c["phys"] == "e2" else (601, 301)
        c["nx"], c["nz"] = size(nxm, 60), size(nzm, 40)
        c["nt"] = size(c["nt"], 120)
        c["shots"] = 1 if c["do"] == "rtm" else rng.randint(1, max(2, c["shots"]))
    c["nrec"] = size(300, 10)
    c["lpml"] = rng.choice([12, 20, 30]) if not c["ny"] else rng.choice([10, 15, 20])
    c["fs"] = rng.random() < 0.3
    if c["do"] in ("call", "plan"):
        c["order"] = rng.choice([8, 8, 8, 6, 4, 5])
    if c["do"] == "fwi":
        c["ncheck"] = rng.choice([10, 20, 40])
        c["ckpt"] = rng.choice(["f16", "bf16"])
    if c["do"] == "rtm":
        c["nhx"] = rng.choice([1, 3, 5])
    return c


# ---------------------------------------------------------------- inputs
def f32(x):
    return float(np.float32(x))


def time_step(c):
    """A time step 10 % under the drivers' stability limit, on a round microsecond."""
    dim = 3 if c["ny"] else 2
    return f32(math.floor(0.9e6 * 2.0 * c["dx"] / (math.pi * math.sqrt(dim) * VMAX)) * 1e-6)


def shot_inputs(c, seed):
    """Per shot: window models, source and receiver positions in cells, the wavelet, and
    for gradients and images the recorded traces."""
    rng = np.random.default_rng([7919, seed])
    dt, dim = time_step(c), 3 if c["ny"] else 2
    f0 = 1500.0 / (7.0 * c["dx"]) if dim == 2 else 1500.0 / (5.0 * c["dx"])
    t = np.arange(c["nt"]) * dt
    out = []
    edges = np.sort(rng.uniform(0.1, 0.9, 5)) * c["nz"]
    speeds = np.linspace(1500.0, 3400.0, 6) * rng.uniform(0.96, 1.04, 6)
    windows = np.random.default_rng(31)      # the survey's apertures, the same for every seed
    for i in range(c["shots"]):
        shape = [c["nz"]]
        for n in (c["ny"], c["nx"]):
            if n:
                shape.append(n if c["shots"] == 1 else max(30, int(n * windows.uniform(0.7, 1.0))))
        z = np.arange(shape[0])
        prof = speeds[np.searchsorted(edges, z)].astype(np.float32)
        vp = np.empty(shape, np.float32)
        vp[:] = prof.reshape((-1,) + (1,) * (dim - 1))
        for _ in range(4):       # smooth seeded anomalies
            g = np.float32(rng.uniform(-0.06, 0.06))
            f = np.ones((1,) * dim, np.float32)
            for a, n in enumerate(shape):
                e = np.exp(-((np.arange(n) - rng.uniform(0.1, 0.9) * n) / (0.12 * n + 4)) ** 2).astype(np.float32)
                f = f * e.reshape((1,) * a + (-1,) + (1,) * (dim - 1 - a))
            vp *= 1 + g * f
        np.minimum(vp, np.float32(VMAX * 0.99), out=vp)
        rho = (np.float32(310.0) * np.sqrt(np.sqrt(vp))).astype(np.float32)
        # horizontal axes last: x = axis -1, y = axis -2 in 3D, z = axis 0; positions (x, [y,] z) in eighths of a cell
        nx, ny = shape[-1], shape[1] if dim == 3 else 0
        eighth = lambda v: np.round(v * 8) / 8  # noqa: E731
        horiz = [eighth(rng.uniform(0.3, 0.7) * n) for n in ((nx, ny) if dim == 3 else (nx,))]
        src = np.array([horiz + [2.0 + 0.125 * rng.integers(0, 8)]])
        if dim == 3:
            m = max(1, math.isqrt(c["nrec"]))
            gx, gy = np.meshgrid(eighth(np.linspace(2, nx - 4, m)), eighth(np.linspace(2, ny - 4, m)))
            rec = np.stack([gx.ravel(), gy.ravel(), np.full(m * m, 1.5)], 1)
        else:
            rec = np.stack([eighth(np.linspace(2, nx - 4, c["nrec"])), np.full(c["nrec"], 1.5)], 1)
        a = (math.pi * f0 * rng.uniform(0.95, 1.05) * (t - 1.0 / f0)) ** 2
        wav = (SOURCE[c["phys"][0]] * (1 - 2 * a) * np.exp(-a)).astype(np.float32)[None]
        s = dict(vp=vp, vs=(vp / np.float32(rng.uniform(1.7, 1.95))).astype(np.float32), rho=rho, src=src, rec=rec,
                 wav=wav)
        if c["do"] in ("fwi", "rtm"):
            # recorded events: hyperbolas with geometric spreading
            r = np.sqrt((((rec - src) * c["dx"]) ** 2).sum(1))[:, None]
            d = np.zeros((len(rec), c["nt"]))
            for _ in range(3):
                t0, v = rng.uniform(0.1, 0.6) * c["nt"] * dt, rng.uniform(1600.0, 2800.0)
                a = (math.pi * f0 * (t[None] - np.sqrt(t0 ** 2 + (r / v) ** 2) - 1.0 / f0)) ** 2
                d += rng.uniform(-1, 1) * (1 - 2 * a) * np.exp(-a) / (1 + r / (20 * c["dx"]))
            s["obs"] = (RECORDED[c["phys"]] * d).astype(np.float32)
        out.append(s)
    return out


# source strengths (volume rate, Pa/s), and the size of a recorded pressure (acoustic) or
# velocity (elastic) sample that they cause
SOURCE = {"a": 1e3, "e": 1e10}
RECORDED = {"a2": 1e8, "e2": 5e-2, "e3": 2e-2}
COMPONENTS = {"a2": ("P",), "a3": ("P",), "e2": ("P", "x", "z"), "e3": ("x", "y", "z")}
FIELD = {"P": abi.PRESSURE, "x": abi.VX, "y": abi.VY, "z": abi.VZ}


def recorded(c, s, comp):
    """Recorded traces of one component (an elastic pressure is an impedance larger)."""
    return (s["obs"] * np.float32(4e6)) if c["phys"] == "e2" and comp == "P" else s["obs"]


def prepare(case, seed):
    c, dt, dim = case, time_step(case), 3 if case["ny"] else 2
    prec = PREC[c["prec"]]
    cls = {"a2": rs.ModelAcoustic2D, "e2": rs.ModelElastic2D, "a3": rs.ModelAcoustic3D, "e3": rs.ModelElastic3D}[c["phys"]]
    data = rs.Data3D if dim == 3 else rs.Data2D
    models, sources, recs = [], [], []

    def traces(pos, field, m, which):
        d = data(len(pos), c["nt"], dt, 0.0, prec)
        (d.scoords if which == rs.SMAP else d.gcoords)[:] = pos * c["dx"]
        d.setField(field)
        d.makeMap(m, which)
        return d

    ins = shot_inputs(c, seed)
    for s in ins:
        n = s["vp"].shape
        size = (n[2], n[1], n[0]) if dim == 3 else (n[1], n[0])
        m = cls(*size, c["lpml"], *(c["dx"],) * dim, *(0.0,) * dim, c["fs"], prec)
        m.createModel()
        m.Vp[:], m.R[:] = s["vp"], s["rho"]
        if c["phys"][0] == "e":
            m.Vs[:] = s["vs"]
        m.staggerModels()
        w = traces(s["src"], abi.PRESSURE, m, rs.SMAP)
        w.data[:] = s["wav"]
        models.append(m)
        sources.append(w)
        if c["do"] in ("call", "plan"):
            recs.append(traces(s["rec"], abi.VX if c["phys"][0] == "e" else abi.PRESSURE, m, rs.GMAP))
        else:
            recs.append([traces(s["rec"], FIELD[k], m, rs.GMAP) for k in COMPONENTS[c["phys"]]])
            for r, k in zip(recs[-1], COMPONENTS[c["phys"]]):
                r.data[:] = recorded(c, s, k)
    state = dict(case=c, models=models, sources=sources, recs=recs)
    if c["do"] == "plan":
        state["plan"] = rs.Plan(models, sources, recs, c["order"], prec)
    if c["do"] == "fwi":
        jobs = []
        for m, w, r in zip(models, sources, recs):
            if c["phys"] == "a2":
                j = rs.FwiAcoustic2D(m, w, r[0], c["order"], 1, prec)
                img = rs.Image2D
            elif c["phys"] == "e2":
                j = rs.FwiElastic2D(m, w, r[0], r[1], r[2], c["order"], 1, prec)
                img = rs.Image2D
            else:
                j = rs.FwiElastic3D(m, w, r[0], r[1], r[2], c["order"], 1, prec)
                img = rs.Image3D
            j.setVpgrad(img("", m))
            j.setRhograd(img("", m))
            if c["phys"][0] == "e":
                j.setVsgrad(img("", m))
            j.setNcheck(c["ncheck"])
            j.setCheckpointPrecision(CKPT[c["ckpt"]])
            j.setAccumulation(abi.ACCUM_F64)
            jobs.append(j)
        state["jobs"], state["batch"] = jobs, rs.AdjointBatch(jobs)
    return state


def grads(job):
    return [getattr(job, k) for k in ("vpgrad", "rhograd", "vsgrad") if getattr(job, k, None) is not None]


def run(state):
    c = state["case"]
    if c["do"] == "plan":
        p = state["plan"]
        p.reset()
        p.run()
        return [p.read_traces(i) for i in range(c["shots"])]
    if c["do"] == "fwi":
        for j in state["jobs"]:
            j.misfit = 0.0
            for g in grads(j):
                g.getImagedata().fill(0)
        state["batch"].run()
        state["batch"].read()
        return [dict(misfit=float(j.misfit), grads=[g.getImagedata() for g in grads(j)]) for j in state["jobs"]]
    if c["do"] == "rtm":
        m = state["models"][0]
        img = rs.Image2D("", m, c["nhx"], 1)
        r = rs.RtmAcoustic2D(m, img, state["sources"][0], state["recs"][0][0], c["order"], 1)
        r.setNcheck(c["ncheck"])
        r.run_optimal()
        return [img.getImagedata()]
    for r in state["recs"]:
        r.data.fill(0)
    if c["shots"] == 1:
        cls = {"a2": rs.ModellingAcoustic2D, "e2": rs.ModellingElastic2D, "a3": rs.ModellingAcoustic3D,
               "e3": rs.ModellingElastic3D}[c["phys"]]
        mod = cls(state["models"][0], state["sources"][0], c["order"])
        (mod.setRecVx if c["phys"][0] == "e" else mod.setRecP)(state["recs"][0])
        mod.run()
    else:
        rs.modelling_batch(state["models"], state["sources"], state["recs"], c["order"], PREC[c["prec"]])
    return [r.data for r in state["recs"]]


# ---------------------------------------------------------------- what a pass cannot do without
def forward_steps(nt, snaps):
    """Forward steps of the binomial checkpoint schedule with `snaps` snapshots."""
    reps = 0
    while math.comb(snaps + reps, snaps) < nt:
        reps += 1
    return nt if reps <= 1 else reps * nt - math.comb(snaps + reps, snaps + 1)


def work(case):
    c, dim = case, 3 if case["ny"] else 2
    fields, params = {"a2": (3, 3), "e2": (5, 5), "a3": (4, 4), "e3": (9, 8)}[c["phys"]]
    derivs = {"a2": 4, "e2": 8, "a3": 6, "e3": 18}[c["phys"]]
    l2, n, strip = 2 * c["lpml"], [c["nx"], c["nz"]] + [c["ny"]] * (dim - 2), 0
    shrink = 1.0 if c["shots"] == 1 else 0.85 ** (dim - 1)      # mean window of a batch
    pts = shrink * math.prod(k + l2 for k in n)
    for k in n:
        strip += pts * l2 / (k + l2) * {"a2": 2, "e2": 4, "a3": 2, "e3": 6}[c["phys"]]
    # per step: every field read and written, every parameter read, the C-PML memory read and written
    step_b, step_f = 4 * (pts * (2 * fields + params) + 2 * strip), pts * derivs * 3 * c["order"]
    steps, extra = c["nt"], 4 * c["nt"] * c["nrec"]
    if c["do"] in ("fwi", "rtm"):
        snaps = c["ncheck"] if c["ncheck"] else int(math.log2(c["nt"])) + 1
        steps = forward_steps(c["nt"], snaps) + c["nt"]
        corr = {"fwi": {"a2": 2, "e2": 3, "e3": 3}.get(c["phys"]), "rtm": c["nhx"]}[c["do"]]
        inner = shrink * math.prod(n)
        extra += c["nt"] * inner * (2 * corr * (8 if c["do"] == "fwi" else 4) + 4 * (2 * fields))
    return {"bytes": float(c["shots"] * (steps * step_b + extra)), "flops": float(c["shots"] * steps * step_f)}


def tolerance(case):
    if case["prec"] == "exact":
        return "exact"       # every operation rounded in the order of the CPU code
    if case["do"] != "fwi":
        # 32-bit sums in another order over a few hundred steps: fused against separately rounded arithmetic
        # differ by up to 4.3e-6 here
        return {"rel": 2e-5}
    # 16-bit checkpoints: the rounding of the saved states dominates (1.8e-4 and 2.2e-3 against lossless ones)
    return {"rel": {"f16": 7e-4, "bf16": 8e-3}[case["ckpt"]]}


# ---------------------------------------------------------------- the same in float64
# staggered-grid coefficients per half-length; shorter stencils stand in near the array ends
COEF = [[], [float(np.float32(1.0029))], [1.188401, -7.046382e-2], [1.216624, -9.197724e-2, 1.300041e-2],
        [1.230862, -1.034123e-1, 2.011671e-2, -3.245760e-3],
        [1.239407, -1.105315e-1, 2.496329e-2, -5.804879e-3, 9.358680e-4],
        [1.245095, -1.153979e-1, 2.848442e-2, -7.899473e-3, 1.898222e-3, -2.935304e-4],
        [1.249150, -1.189375e-1, 3.116091e-2, -9.623004e-3, 2.812069e-3, -6.655106e-4, 9.728191e-5],
        [1.252186, -1.216289e-1, 3.326513e-2, -1.105777e-2, 3.647865e-3, -1.066144e-3, 2.437491e-4, -3.351959e-5]]


def banded(n, order, d, forward, dev):
    m = np.zeros((n, n))
    for i in range(n):
        k = min(order, i + 1, n - 1 - i) if forward else min(order, i, n - i)
        for j in range(max(k, 0)):
            hi, lo = (i + j + 1, i - j) if forward else (i + j, i - j - 1)
            m[i, hi] += COEF[k][j] / d
            m[i, lo] -= COEF[k][j] / d
    return torch.from_numpy(m).to(dev)


def absorbing(n, lpml, dt, half):
    """C-PML factors A, B, C along an axis of n cells (half: at the half cells)."""
    out = np.zeros((3, n))
    for i in range(lpml):
        for x, at in (((lpml - i - half) / lpml, i), ((i + 1.0 + half) / lpml, n - lpml + i)):
            g = x ** 3
            k, s = 1.0 + g, 1200.0 * g
            b = math.exp(-s / k * dt)
            out[:, at] = (s * (1.0 - b) / (k * s), b, 1.0 - 1.0 / k)
    return out


class Shot64:
    """One shot's wavefields in float64, axes "x", "y", "z" (array axes -1, -2, 0)."""

    def __init__(self, c, s, dev):
        self.c, self.dev, self.dt, self.l = c, dev, time_step(c), c["lpml"]
        self.elastic, self.axes = c["phys"][0] == "e", "xyz" if c["ny"] else "xz"
        pad = lambda a: torch.from_numpy(np.pad(a, self.l, mode="edge").astype(np.float64)).to(dev)  # noqa: E731
        vp, vs, rho = pad(s["vp"]), pad(s["vs"]), pad(s["rho"])
        self.shape = vp.shape
        self.n = {a: vp.shape[self.at(a)] for a in self.axes}
        d = f32(c["dx"])
        self.D = {(a, f): banded(self.n[a], c["order"], d, f, dev) for a in self.axes for f in (True, False)}
        self.pml = {}
        for a in self.axes:
            for f in (True, False):
                t = torch.from_numpy(absorbing(self.n[a], self.l, self.dt, 0.5 if f else 0.0)).to(dev)
                view = [1] * len(self.shape)
                view[self.at(a)] = -1
                self.pml[a, f] = [q.reshape(view) for q in t]
        self.vp, self.vs, self.rho = (self.inner(q) for q in (vp, vs, rho))
        self.R = {a: 1.0 / self.average(rho, a) for a in self.axes}
        if self.elastic:
            mu = rho * vs * vs
            self.L2M, self.L = rho * vp * vp, rho * vp * vp - 2.0 * mu
            self.M = {a + b: self.average(self.average(mu, a), b) for a in self.axes for b in self.axes if a < b}
            if c["fs"]:
                self.L[self.l], self.L2M[self.l] = 0.0, mu[self.l]
        else:
            self.L = rho * vp * vp
            if c["fs"]:
                self.L[self.l] = 0.0
        if c["fs"]:
            for a in self.axes[:-1]:
                self.R[a][self.l] *= 2.0
        self.clear()

    def at(self, a):
        return {"x": -1, "y": -2, "z": 0}[a]

    def average(self, m, a):
        k = self.at(a) % m.dim()
        mean = 0.5 * (m.narrow(k, 1, m.shape[k] - 1) + m.narrow(k, 0, m.shape[k] - 1))
        return torch.cat([mean, mean.narrow(k, mean.shape[k] - 1, 1)], k)

    def clear(self):
        zero = lambda: torch.zeros(self.shape, dtype=torch.float64, device=self.dev)  # noqa: E731
        self.psi, self.V = {}, {a: zero() for a in self.axes}
        names = [a + b for a in self.axes for b in self.axes if a <= b] if self.elastic else ["P"]
        self.S = {k: zero() for k in names}

    def deriv(self, f, a, forward, key):
        m = self.D[a, forward]
        if a == "x":
            d = f @ m.T
        elif a == "y":
            d = torch.matmul(m, f)
        else:
            d = (m @ f.reshape(f.shape[0], -1)).reshape(f.shape)
        A, B, C = self.pml[a, forward]
        self.psi[key] = A * d if key not in self.psi else B * self.psi[key] + A * d
        return d - self.psi[key] - C * d

    def step(self, adjoint=False):
        dt, S, V = self.dt, self.S, self.V
        if not self.elastic:
            for a in self.axes:
                V[a] += dt * self.R[a] * self.deriv(S["P"], a, True, "v" + a)
            for a in self.axes:
                S["P"] += dt * self.L * self.deriv(V[a], a, False, "p" + a)
            return
        W = S
        if adjoint:
            tr = sum(S[a + a] for a in self.axes)
            W = {k: self.L * tr + (self.L2M - self.L) * S[k] if k[0] == k[1] else self.M[k] * S[k] for k in S}
        for a in self.axes:
            V[a] += dt * self.R[a] * sum(self.deriv(W[min(a, b) + max(a, b)], b, a == b, "v" + a + b) for b in self.axes)
        e = {a: self.deriv(V[a], a, False, "n" + a) for a in self.axes}
        tr = sum(e.values())
        for a in self.axes:
            S[a + a] += dt * (e[a] if adjoint else self.L * tr + (self.L2M - self.L) * e[a])
        if self.c["fs"]:
            S["zz"][self.l] = 0.0
        for k in (q for q in S if q[0] != q[1]):
            d = self.deriv(V[k[0]], k[1], True, "s" + k + k[1]) + self.deriv(V[k[1]], k[0], True, "s" + k + k[0])
            S[k] += dt * (d if adjoint else self.M[k] * d)

    def points(self, pos, comp):
        """Flat indices [n, corners] and weights of positions (x, [y,] z) in cells."""
        n = len(pos)
        idx, w = np.zeros((n, 1), np.int64), np.ones((n, 1))
        for j, a in enumerate(self.axes):
            p = pos[:, j] - (0.5 if comp == a else 0.0)
            i = np.floor(p).astype(np.int64)
            stride = {"x": 1, "y": self.n["x"], "z": int(np.prod(self.shape[1:]))}[a]
            cell = (i + self.l)[:, None] * stride + np.array([0, stride])
            share = np.stack([1 - (p - i), p - i], 1)
            idx = (idx[:, :, None] + cell[:, None, :]).reshape(n, -1)
            w = (w[:, :, None] * share[:, None, :]).reshape(n, -1)
        return torch.from_numpy(idx).to(self.dev), torch.from_numpy(w).to(self.dev)

    def inject(self, pts, comp, w):
        idx, wt = pts
        v, idx = (wt * w[:, None]).reshape(-1), idx.reshape(-1)
        add = lambda f, x: f.view(-1).index_add_(0, idx, x)  # noqa: E731
        if comp != "P":
            add(self.V[comp], self.dt * self.R[comp].reshape(-1)[idx] * v)
        elif self.elastic:
            for a in self.axes:
                add(self.S[a + a], -self.dt * v)
        else:
            add(self.S["P"], self.dt * self.L.reshape(-1)[idx] * v)

    def record(self, pts, comp):
        idx, wt = pts
        if comp != "P":
            f = self.V[comp]
        elif self.elastic:
            f = sum(self.S[a + a] for a in self.axes) / len(self.axes)
        else:
            f = self.S["P"]
        return (wt * f.reshape(-1)[idx]).sum(1)

    def inner(self, f, **off):
        """The unpadded window of f, shifted by off cells along its axes."""
        for a in self.axes:
            f = f.narrow(self.at(a) % f.dim(), self.l + off.get(a, 0), self.n[a] - 2 * self.l)
        return f


def forward64(p, s, c, comps, keep):
    src = p.points(s["src"], "P")
    rec = [p.points(s["rec"], k) for k in comps]
    wav = torch.from_numpy(s["wav"].astype(np.float64)).to(p.dev)
    out = [torch.zeros(len(s["rec"]), c["nt"], dtype=torch.float64, device=p.dev) for _ in comps]
    states = []
    for it in range(c["nt"]):
        p.step()
        p.inject(src, "P", wav[:, it])
        for o, r, k in zip(out, rec, comps):
            o[:, it] = p.record(r, k)
        if keep and p.elastic:
            states.append(({a: v.clone() for a, v in p.V.items()}, {a: v.clone() for a, v in p.S.items()}))
        elif keep:
            states.append(p.S["P"].clone())
    return out, states


def gradient64(p, s, c):
    comps = COMPONENTS[c["phys"]]
    mod, states = forward64(p, s, c, comps, True)
    res = [m - torch.from_numpy(recorded(c, s, k).astype(np.float64)).to(p.dev) for m, k in zip(mod, comps)]
    misfit = float(sum((0.5 * r * r).sum() for r in res))
    rec = [p.points(s["rec"], k) for k in comps]
    p.clear()
    g = [torch.zeros_like(p.inner(p.R["x"])) for _ in range(3)]
    for it in range(c["nt"] - 1, -1, -1):
        last = it == c["nt"] - 1
        if not last:
            p.step(adjoint=True)
        for q, k, r in zip(rec, comps, res):
            p.inject(q, k, r[:, it])
        if it > 0:     # the adjoint time it meets the forward state before step it, the last one its own
            correlate64(p, states[it if last else it - 1], c, g)
            states[it] = None
    vp, vs, rho = p.vp, p.vs, p.rho
    if not p.elastic:
        return misfit, [g[0], g[1]]
    lam, mu, r = g
    last = r + vs * vs * mu + (vp * vp - (0 if c["ny"] else 2) * vs * vs) * lam
    return misfit, [2 * rho * vp * lam, last, 2 * rho * vs * mu - 4 * rho * vs * lam]


def correlate64(p, fwd, c, g):
    """One adjoint time's contribution to the gradients, on the interior of the window."""
    h = f32(c["dx"])
    win = p.inner
    cut = tuple(slice(1, -1) for _ in p.axes)
    if not p.elastic:
        f, sdiv, ud = win(fwd), 0, 0
        for a in p.axes:
            v, r = p.V[a], p.R[a]
            sdiv = sdiv + (win(v) - win(v, **{a: -1})) / h
            up = win(v) * win(r) * (win(fwd, **{a: 1}) - f)
            dn = win(v, **{a: -1}) * win(r, **{a: -1}) * (f - win(fwd, **{a: -1}))
            ud = ud + 0.5 * (up + dn) / h
        g[0][cut] += (2 / p.vp * f * sdiv)[cut]
        g[1][cut] += (1 / p.rho * f * sdiv + ud)[cut]
        return
    V, S = fwd
    A = p.S
    m = {a: (win(V[a]) - win(V[a], **{a: -1})) / h for a in p.axes}
    g[0][cut] -= (sum(m.values()) * sum(win(A[a + a]) for a in p.axes))[cut]

    def corner(a, b, oa, ob):
        # strain of the shear pair (a, b) at the corner whose upper ends are oa, ob cells away
        x = win(V[b], **{a: oa, b: ob - 1}) - win(V[b], **{a: oa - 1, b: ob - 1})
        y = win(V[a], **{a: oa - 1, b: ob}) - win(V[a], **{a: oa - 1, b: ob - 1})
        return (x + y) / h

    if len(p.axes) == 2:
        t = 2 * (m["x"] * win(A["zz"]) + m["z"] * win(A["xx"]))
        t = t - 0.25 * sum(corner("x", "z", i, j) * win(A["xz"], x=i - 1, z=j - 1) for i in (0, 1) for j in (0, 1))
        g[1][cut] += t[cut]
    else:
        t = 2 * sum(m[a] * win(A[a + a]) for a in p.axes)
        for a, b in ("yz", "xz", "xy"):
            t = t + 0.25 * sum(corner(a, b, i, j) for i in (0, 1) for j in (0, 1)) * win(A[a + b])
        g[1][cut] -= t[cut]
    rh = 0
    for a in p.axes:
        v, r = p.V[a], p.R[a]
        # stress divergence on the face above, and on the face below along a; in 3D the CPU
        # code weights the lower z face with the adjoint Vz of the cell at y-1
        low = win(v, y=-1) if a == "z" and len(p.axes) == 3 else win(v, **{a: -1})
        for at, wgt in ((0, win(v) * win(r)), (-1, low * win(r, **{a: -1}))):
            div = 0
            for b in p.axes:
                f = S[min(a, b) + max(a, b)]
                up, dn = ({a: at + 1}, {a: at}) if b == a else ({a: at}, {a: at, b: -1})
                div = div + (win(f, **up) - win(f, **dn)) / h
            rh = rh + 0.5 * wgt * div
    g[2][cut] -= rh[cut]


def exact(case, seed):
    c = case
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    out = []
    for s in shot_inputs(c, seed):
        p = Shot64(c, s, dev)
        if c["do"] in ("call", "plan"):
            d, _ = forward64(p, s, c, ("x",) if p.elastic else ("P",), False)
            out.append(d[0].cpu().numpy())
        elif c["do"] == "fwi":
            mis, g = gradient64(p, s, c)
            dims = (1, 1, 1) if c["ny"] else (1, 1)
            out.append(dict(misfit=mis, grads=[x.reshape(dims + tuple(x.shape)).cpu().numpy() for x in g]))
        else:
            _, states = forward64(p, s, c, (), True)
            obs, rec = torch.from_numpy(s["obs"].astype(np.float64)).to(dev), p.points(s["rec"], "P")
            p.clear()
            nx, img = c["nx"], torch.zeros(1, c["nhx"], c["nz"], c["nx"], dtype=torch.float64, device=dev)
            for it in range(c["nt"] - 1, -1, -1):
                last = it == c["nt"] - 1
                if not last:
                    p.step()
                p.inject(rec, "P", obs[:, it])
                if it == 0:
                    continue
                f, b = p.inner(states[it if last else it - 1]), p.inner(p.S["P"])
                for k in range(c["nhx"]):
                    h = abs(k - (c["nhx"] - 1) // 2)
                    i = slice(h, nx - h)
                    lo, hi = slice(0, nx - 2 * h), slice(2 * h, nx)
                    fs, bs = (lo, hi) if k >= (c["nhx"] - 1) // 2 else (hi, lo)
                    img[0, k][:, i] += f[:, fs] * b[:, bs]
            out.append(img.cpu().numpy())
    return out
