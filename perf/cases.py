"""The work that users of this framework have it do, as measurable cases.

A pass is a whole job through the public entry points, as a host program
runs it between two save events: upload a state in VAC's layout from
page-locked host memory, advance it some time steps, take the new state
back.  Three kinds of job:

* ``engine``: one grid through ``Engine`` (upload_flat, step, download_flat);
* ``batch``: many uneven grids through ``Batch`` and the batch calls of the
  C ABI, every grid its own run;
* ``server``: requests of mixed sizes and step counts submitted to
  ``Server`` and collected.

Sizes, problems and options are those of the configurations, the benchmark
and the tests: Orszag-Tang-like vortices, random Fourier modes, blasts with
outflow, two-state Riemann problems, shock tubes; FP64 and the mixed
precision path, TVDLF and the Roe dissipation ('tvdmu'), minmod and woodward
limiters, periodic and outflow faces.  The state of a mixed run lives in FP32
on the device, so such a job keeps its result as float32; an FP64 run keeps
float64.

``exact`` advances the same state in float64 with whole-array torch
operations (TVDLF/Hancock and the eight-wave Roe solver written out below,
without this repository's code).
"""
import ctypes as C
import math

import numpy as np
import torch

from vac_gb300 import abi, engine

# --------------------------------------------------------------- the cases


def _engine(name, physics, nx, init, steps, precision, limiter="minmod", bc="periodic",
            method="tvdlf", p0=0.05):
    c = {"job": "engine", "physics": physics, "ndim": len(nx), "init": init, "steps": steps,
         "precision": precision, "limiter": limiter, "bc": bc, "method": method, "p0": p0}
    for d, n in enumerate(nx):
        c["n%d" % (d + 1)] = int(n)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # VAC's shock-tube run: 1-D gas, one hundred cells; nothing but
        # launches and their latency
        _engine("tube100_fp64", "hd", (100,), "tube", 100, "fp64", bc="cont"),
        # the plain configuration: Orszag-Tang on 200^2, 200 steps in FP64
        _engine("vortex200_fp64", "mhd", (200, 200), "vortex", 200, "fp64"),
        # a 3-D blast in FP64 with outflow on a ragged grid: the parity path
        # at the size where the FP64 pipe decides
        _engine("blast96_fp64", "mhd", (96, 101, 90), "blast", 10, "fp64", "woodward", "cont"),
        # the Roe dissipation in FP64 on a 2-D vortex (the tests' tvdmu runs)
        _engine("vortex_roe_fp64", "mhd", (160, 144), "vortex", 40, "fp64", "woodward",
                method="tvdmu"),
        # the Roe dissipation on the mixed path, 3-D, ragged
        _engine("modes_roe_mixed", "mhd", (128, 113, 120), "modes", 20, "mixed", "woodward",
                method="tvdmu", p0=0.5),
        # the smallest served grids: 128^2 and 64^3, many steps each
        _engine("modes128sq_mixed", "mhd", (128, 128), "modes", 100, "mixed", p0=0.5),
        _engine("modes64_mixed", "mhd", (64, 64, 64), "modes", 60, "mixed", "woodward", p0=0.5),
        # a served 2-D grid of ordinary size, odd sides
        _engine("modes1001sq_mixed", "mhd", (1001, 962), "modes", 60, "mixed", p0=0.5),
        # the headline configuration: 256^3 low-beta modes, woodward, mixed
        _engine("modes256_mixed", "mhd", (256, 256, 256), "modes", 40, "mixed", "woodward"),
        # the large blast with outflow faces, mixed
        _engine("blast320_mixed", "mhd", (320, 320, 320), "blast", 20, "mixed", "woodward",
                "cont"),
        # the batched configuration: 64 uneven 2-D gas grids, 50 steps each
        {"name": "riemann64_mixed", "job": "batch", "grids": 64, "lo": 64, "hi": 1024,
         "steps": 50, "limiter": "minmod"},
        # the served stream: 2-D and 3-D requests of mixed sizes and lengths
        {"name": "served12_mixed", "job": "server", "requests": 12, "lo2": 128, "hi2": 700,
         "lo3": 64, "hi3": 112, "smin": 20, "smax": 100},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _ragged(rng, side, ndim):
    return tuple(max(8, int(round(side * rng.uniform(0.85, 1.15)))) for _ in range(ndim))


# (weight, physics, ndim, init, precision, method, least and largest side,
#  cell updates and steps a pass has at most): the families of single grids
_FAMILIES = [
    (1, "hd", 1, "tube", "fp64", "tvdlf", 64, 2000, 1e6, 150),
    (2, "mhd", 2, "vortex", "fp64", "tvdlf", 48, 320, 8e6, 200),
    (1, "hd", 2, "riemann", "fp64", "tvdlf", 48, 400, 8e6, 150),
    (2, "mhd", 3, "blast", "fp64", "tvdlf", 32, 100, 8e6, 40),
    (1, "mhd", 2, "vortex", "fp64", "tvdmu", 48, 180, 9e5, 60),
    (2, "mhd", 3, "modes", "mixed", "tvdmu", 40, 140, 3.4e7, 40),
    (1, "mhd", 2, "modes", "mixed", "tvdmu", 64, 600, 2e7, 80),
    (2, "mhd", 2, "modes", "mixed", "tvdlf", 96, 1600, 6e7, 120),
    (1, "hd", 2, "riemann", "mixed", "tvdlf", 64, 1200, 6e7, 120),
    (3, "mhd", 3, "modes", "mixed", "tvdlf", 48, 260, 4e8, 80),
    (2, "mhd", 3, "blast", "mixed", "tvdlf", 48, 260, 4e8, 60),
]


def draw(rng):
    kind = rng.random()
    if kind < 0.08:
        lo = _logint(rng, 48, 160)
        return {"job": "batch", "grids": rng.randint(8, 64), "lo": lo,
                "hi": _logint(rng, 4 * lo, 1024), "steps": rng.randint(10, 50),
                "limiter": rng.choice(["minmod", "woodward"])}
    if kind < 0.16:
        return {"job": "server", "requests": rng.randint(4, 12), "lo2": _logint(rng, 64, 160),
                "hi2": _logint(rng, 320, 700), "lo3": _logint(rng, 40, 64),
                "hi3": _logint(rng, 72, 112), "smin": rng.randint(4, 20),
                "smax": rng.randint(40, 100)}
    f = rng.choices(_FAMILIES, [f[0] for f in _FAMILIES])[0]
    _, physics, ndim, init, precision, method, lo, hi, most, msteps = f
    nx = _ragged(rng, _logint(rng, lo, hi), ndim)
    steps = max(4, min(msteps, int(most / np.prod(nx, dtype=float))))
    steps = rng.randint(max(4, steps // 2), steps)
    bc = "cont" if init in ("tube", "riemann", "blast") else "periodic"
    return _engine(None, physics, nx, init, steps, precision, rng.choice(["minmod", "woodward"]),
                   bc, method, p0=0.5 if init == "modes" else 0.05)


def _nx(c):
    return tuple(c["n%d" % (d + 1)] for d in range(c["ndim"]))


def _nw(physics, ndim):
    return 2 + 2 * ndim if physics == "mhd" else 2 + ndim


# ------------------------------------------------------------ initial states
# Meshes are held as (..., n3, n2, n1) so that a flat view is VAC's order
# (x fastest); component d lies along axis -1-d.


def _axes(nx, lo, hi):
    out = []
    for d, n in enumerate(nx):
        h = (hi - lo) / n
        x = lo + h * (torch.arange(n, dtype=torch.float64) + 0.5)
        shape = [1] * len(nx)
        shape[len(nx) - 1 - d] = n
        out.append(x.reshape(shape).cuda())
    return out


def _wavevectors(rng, count, ndim):
    ks = []
    while len(ks) < count:
        k = rng.integers(-4, 5, size=3)
        k[ndim:] = 0
        if 0 < int((k * k).sum()) <= 16:
            ks.append(k.astype(float))
    return ks


def _cosines(rng, X, ks):
    return [torch.cos(2 * math.pi * sum(float(k[d]) * X[d] for d in range(len(X)) if k[d])
                      + float(rng.uniform(0, 2 * math.pi))) for k in ks]


def _state(physics, nx, init, p0, seed):
    """(mesh coordinate arrays along each axis, conservative state, dx)."""
    rng = np.random.default_rng(seed)
    nd = len(nx)
    lo, hi = {"vortex": (0.0, 2 * math.pi), "blast": (-0.5, 0.5)}.get(init, (0.0, 1.0))
    X = _axes(nx, lo, hi)
    full = tuple(reversed(nx))
    one = torch.ones(full, dtype=torch.float64, device="cuda")
    zero = torch.zeros_like(one)
    gamma = 1.4 if physics == "hd" else 5.0 / 3.0
    b = []
    if init == "tube":
        left = X[0] < rng.uniform(0.4, 0.6)
        rho = torch.where(left, one, one * rng.uniform(0.1, 0.3))
        p = torch.where(left, one, one * rng.uniform(0.08, 0.2))
        v = [zero]
    elif init == "riemann":
        px, py = rng.uniform(0.2, 0.8, 2)
        ang = rng.uniform(0, math.pi)
        left = ((X[0] - px) * math.sin(ang) - (X[1] - py) * math.cos(ang)) < 0
        st = []
        for _ in range(2):
            r, q = rng.uniform(0.1, 1.0, 2)
            th, sp = rng.uniform(0, 2 * math.pi), rng.uniform(0, 0.5)
            st.append((r, q, sp * math.cos(th), sp * math.sin(th)))
        pick = [torch.where(left, one * a, one * c) for a, c in zip(*st)]
        rho, p, v = pick[0], pick[1], pick[2:]
    elif init == "vortex":
        f = rng.uniform(0, 2 * math.pi, 4)
        rho, p = one * gamma * gamma, one * gamma
        v = [-torch.sin(X[1] + f[0]) * one, torch.sin(X[0] + f[1]) * one]
        b = [-torch.sin(X[1] + f[2]) * one, torch.sin(2 * X[0] + f[3]) * one]
    elif init == "blast":
        c = rng.uniform(-0.1, 0.1, nd)
        r = torch.sqrt(sum((X[d] - c[d]) ** 2 for d in range(nd)))
        p = 0.1 + 9.9 * 0.5 * (1 - torch.tanh((r - 0.1) / (1.0 / max(nx))))
        th = rng.uniform(0, 2 * math.pi)
        rho, v = one, [zero] * nd
        b = [one * math.cos(th), one * math.sin(th)] + [zero] * (nd - 2)
    else:  # random Fourier modes around a uniform field along x
        a = rng.uniform(0.5, 1.0, 8)
        a *= 0.2 / a.sum()
        rho = one.clone()
        for ak, cs in zip(a, _cosines(rng, X, _wavevectors(rng, 8, nd))):
            rho += float(ak) * cs
        dirs = rng.normal(size=(8, 3))
        cs = _cosines(rng, X, _wavevectors(rng, 8, nd))
        v = [sum(float(dirs[i, d]) * cs[i] for i in range(8)) * one for d in range(nd)]
        rms = float(torch.sqrt(sum(t * t for t in v).mean()))
        v = [t * (0.3 / rms) for t in v]
        ks = _wavevectors(rng, 8, nd)
        pol = [np.cross(rng.normal(size=3), k) for k in ks]
        cs = _cosines(rng, X, ks)
        b = [sum(float(pol[i][d]) * cs[i] for i in range(8)) * one for d in range(nd)]
        rms = float(torch.sqrt(sum(t * t for t in b).mean()))
        b = [t * (0.1 / rms) for t in b]
        b[0] = b[0] + 1.0
        p = one * p0
    e = p / (gamma - 1) + 0.5 * rho * sum(t * t for t in v)
    if b:
        e = e + 0.5 * sum(t * t for t in b)
    w = torch.stack([t.expand(full) for t in [rho] + [rho * t for t in v] + [e] + b])
    x = torch.stack([t.expand(full) for t in X])
    return x, w, [(hi - lo) / n for n in nx], gamma


def _params(physics, nx, gamma, limiter, bc, precision, method):
    nd = len(nx)
    p = abi.default_params(nd, nd, abi.PHYS_MHD if physics == "mhd" else abi.PHYS_HD, list(nx),
                           gamma=gamma)
    p.typefull = abi.TYPEFULL_NAMES[method]
    p.precision = abi.PREC_MIXED if precision == "mixed" else abi.PREC_FP64
    abi.set_all_limiters(p, abi.LIMITER_NAMES[limiter])
    abi.set_all_bc(p, abi.BC_NAMES[bc])
    return p


def _fortran(a):
    """A (k, n3, n2, n1) tensor as numpy (k, n1, n2, n3) without a copy."""
    a = a.numpy()
    return a.transpose((0,) + tuple(range(a.ndim - 1, 0, -1)))


def _pinned(n, dtype=torch.float64):
    return torch.empty(n, dtype=dtype, pin_memory=True)


# ---------------------------------------------------------- prepare and run


def _batch_grids(c, seed):
    rng = np.random.default_rng(c["lo"] * 4096 + c["hi"])  # the sides belong to the case
    sides = [int(round(v)) for v in np.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"]),
                                                       c["grids"]))]
    return [("hd", (s, s), "riemann", c["steps"], 0.05, seed * 1000 + i)
            for i, s in enumerate(sides)]


def _server_grids(c, seed):
    rng = np.random.default_rng(c["lo2"] * 4096 + c["hi3"])
    out = []
    for i in range(c["requests"]):
        nd = 2 if i % 2 == 0 else 3
        lo, hi = (c["lo2"], c["hi2"]) if nd == 2 else (c["lo3"], c["hi3"])
        side = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        out.append(("mhd", (side,) * nd, "modes", int(rng.integers(c["smin"], c["smax"] + 1)),
                    0.5, seed * 1000 + i))
    return out


def prepare(case, seed):
    c = dict(case)
    if c["job"] == "engine":
        nx = _nx(c)
        x, w, _, gamma = _state(c["physics"], nx, c["init"], c["p0"], seed)
        src = _pinned(w.numel())
        src.copy_(w.reshape(-1))
        p = _params(c["physics"], nx, gamma, c["limiter"], c["bc"], c["precision"], c["method"])
        e = engine.Engine(p, _fortran(x.cpu()), _fortran(src.reshape(w.shape)))
        s = {"job": "engine", "engine": e, "src": src, "dst": _pinned(w.numel()),
             "steps": c["steps"]}
        if c["precision"] == "mixed":
            s["single"] = torch.zeros(w.numel(), dtype=torch.float32)
        return s
    specs = _batch_grids(c, seed) if c["job"] == "batch" else _server_grids(c, seed)
    grids, parts = [], []
    for physics, nx, init, steps, p0, sd in specs:
        x, w, _, gamma = _state(physics, nx, init, p0, sd)
        p = _params(physics, nx, gamma, c.get("limiter", "minmod" if len(nx) == 2 else "woodward"),
                    "cont" if c["job"] == "batch" else "periodic", "mixed", "tvdlf")
        grids.append((p, x.cpu(), steps))
        parts.append(w.reshape(-1))
    n = sum(t.numel() for t in parts)
    src, at = _pinned(n), []
    o = 0
    for t in parts:
        src[o:o + t.numel()].copy_(t)
        at.append(o)
        o += t.numel()
    s = {"job": c["job"], "src": src, "dst": _pinned(n), "at": at, "n": len(grids),
         "single": torch.zeros(n, dtype=torch.float32), "t": torch.zeros(len(grids))}
    if c["job"] == "batch":
        s["batch"] = engine.Batch([(p, _fortran(x), _fortran(t.cpu().reshape((-1,) + x.shape[1:])))
                                   for (p, x, _), t in zip(grids, parts)])
        s["steps"] = c["steps"]
    else:
        s["server"] = engine.Server(hbm_budget_bytes=150e9, max_active=8, steps_per_chunk=16)
        flat = src.numpy()
        ends = at[1:] + [n]
        s["requests"] = [(p, x.reshape(-1).numpy(), flat[a:z], steps)
                         for (p, x, steps), a, z in zip(grids, at, ends)]
    return s


def _check(rc):
    if rc:
        raise RuntimeError(engine.last_error())


def _at(buf, offset):
    return C.cast(buf.data_ptr() + 8 * offset, C.POINTER(C.c_double))


def run(s):
    if s["job"] == "engine":
        e = s["engine"]
        e.upload_flat(s["src"].data_ptr())
        e.step(s["steps"])
        e.download_flat(s["dst"].data_ptr())
        if "single" in s:  # dt of a mixed run follows from FP32 wave speeds
            return {"w": s["single"].copy_(s["dst"]), "t": np.float32(e.t), "it": e.it}
        return {"w": s["dst"], "t": np.float64(e.t), "it": e.it}
    L, src, dst, t = engine.lib(), s["src"], s["dst"], s["t"]
    if s["job"] == "batch":
        b = s["batch"]
        for i, o in enumerate(s["at"]):
            _check(L.vacgpu_batch_upload(b.h, i, _at(src, o), 0, 0.0))
        b.step(s["steps"])
        for i, o in enumerate(s["at"]):
            _check(L.vacgpu_batch_download(b.h, i, _at(dst, o)))
            t[i] = b.status(i)[0]
    else:
        srv = s["server"]
        ids = [srv.submit(*r) for r in s["requests"]]
        ts, it, tts = C.c_double(), C.c_int(), C.c_double()
        for i, (rid, o) in enumerate(zip(ids, s["at"])):
            rc = 1
            while rc == 1:
                rc = L.vacgpu_server_result(srv.h, rid, 10.0, _at(dst, o), C.byref(ts),
                                            C.byref(it), C.byref(tts))
            _check(rc)
            t[i] = ts.value
    return {"w": s["single"].copy_(dst), "t": t}


# ------------------------------------------------------------------- work

# Operations of one cell in one sweep: the predictor's two fluxes, the face's
# two and its fast speed (or Roe's waves), slopes, update and sources
_FLOPS = {("hd", "tvdlf"): 180, ("mhd", "tvdlf"): 420, ("mhd", "tvdmu"): 900}


def work(case):
    c = dict(case)
    if c["job"] == "engine":
        jobs = [(c["physics"], _nx(c), c["steps"], c["method"], 8 if c["precision"] == "fp64"
                 else 4)]
    else:
        specs = _batch_grids(c, 0) if c["job"] == "batch" else _server_grids(c, 0)
        jobs = [(ph, nx, steps, "tvdlf", 4) for ph, nx, _, steps, _, _ in specs]
    nbytes = flops = 0.0
    for ph, nx, steps, method, size in jobs:
        cells = float(np.prod(nx, dtype=float))
        values = cells * _nw(ph, len(nx))
        # host state in and out (8 bytes a value), and the state once read
        # and once written in each time step
        nbytes += 2 * 8 * values + 2 * size * values * steps
        flops += cells * steps * len(nx) * _FLOPS[ph, method]
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------- the same in float64, torch


class _Scheme:
    """VAC's split two-step Hancock/TVDLF scheme (or TVD-MUSCL with the
    eight-wave Roe solver) on a uniform grid, on (nw, ..., n2, n1) arrays."""

    def __init__(self, physics, dx, gamma, limiter, bc, method):
        self.mhd, self.dx, self.g = physics == "mhd", dx, gamma
        self.nd = len(dx)
        self.limiter, self.bc, self.roe = limiter, bc, method == "tvdmu"
        self.E = self.nd + 1

    def pad(self, w):
        for d in range(self.nd):
            ax, n = w.dim() - 1 - d, w.shape[w.dim() - 1 - d]
            if self.bc == "periodic":
                w = torch.cat([w.narrow(ax, n - 2, 2), w, w.narrow(ax, 0, 2)], ax)
            else:
                a, z = w.narrow(ax, 0, 1), w.narrow(ax, n - 1, 1)
                w = torch.cat([a, a, w, z, z], ax)
        return w

    def cut(self, W, d, lo, n):
        """Mesh cells in the other directions, cells lo.. of direction d (0
        is the first ghost layer)."""
        for k in range(self.nd):
            ax = W.dim() - 1 - k
            W = W.narrow(ax, lo, n) if k == d else W.narrow(ax, 2, W.shape[ax] - 4)
        return W

    def limit(self, a, b):
        s = torch.copysign(torch.ones_like(a), a)
        m = torch.minimum(a.abs(), s * b)
        if self.limiter == "woodward":
            m = torch.minimum(m, 0.25 * s * (a + b))
            return 2 * s * m.clamp(min=0)
        return s * m.clamp(min=0)

    def m(self, u):
        return u[1:1 + self.nd]

    def b(self, u):
        return u[self.E + 1:self.E + 1 + self.nd]

    def pressure(self, u):
        q = (self.m(u) ** 2).sum(0) / u[0]
        if self.mhd:
            q = q + (self.b(u) ** 2).sum(0)
        return (self.g - 1) * (u[self.E] - 0.5 * q)

    def flux(self, u, d):
        v, p = u[1 + d] / u[0], self.pressure(u)
        f = v * u
        if self.mhd:
            b = self.b(u)
            pt = p + 0.5 * (b ** 2).sum(0)
            f[1:1 + self.nd] -= b * b[d]
            f[1 + d] += pt
            f[self.E] += (u[1 + d] * pt - b[d] * (b * self.m(u)).sum(0)) / u[0]
            f[self.E + 1:] -= self.m(u) / u[0] * b[d]
            f[self.E + 1 + d] = 0
        else:
            f[1 + d] += p
            f[self.E] += v * p
        return f

    def cmax(self, u, d):
        cs2 = self.g * self.pressure(u) / u[0]
        v = (u[1 + d] / u[0]).abs()
        if not self.mhd:
            return cs2.sqrt() + v
        b = self.b(u)
        cf2 = (b ** 2).sum(0) / u[0] + cs2
        q = (cf2 ** 2 - 4 * cs2 * b[d] ** 2 / u[0]).clamp(min=0).sqrt()
        return (0.5 * (cf2 + q)).sqrt() + v

    def powell(self, W, u, qdt, out):
        if not self.mhd:
            return out
        div = 0
        for d in range(self.nd):
            B, n = W[self.E + 1 + d:self.E + 2 + d], u.shape[u.dim() - 1 - d]
            div = div + (self.cut(B, d, 3, n) - self.cut(B, d, 1, n))[0] / (2 * self.dx[d])
        q, b, m = qdt * div, self.b(u), self.m(u)
        out[1:1 + self.nd] -= q * b
        out[self.E + 1:] -= q * m / u[0]
        out[self.E] -= q * (m * b).sum(0) / u[0]
        return out

    def waves(self, L, R, d):
        """sum over waves of |a| (l dw) r, and max |v + cf|, |v - cf|."""
        nd, E, g = self.nd, self.E, self.g
        rL, rR = L[0], R[0]
        rho = 0.5 * (rL + rR)
        vL, vR = self.m(L) / rL, self.m(R) / rR
        v, B = 0.5 * (vL + vR), 0.5 * (self.b(L) + self.b(R))
        vd, bd = v[d], B[d]
        dw = R - L
        db, dv = self.b(dw), vR - vL
        p = 0.5 * (self.pressure(L) + self.pressure(R))
        dp = (g - 1) * (dw[E] - (v * self.m(dw)).sum(0) + 0.5 * (v ** 2).sum(0) * dw[0]
                        - 0.5 * ((self.b(R) ** 2) - (self.b(L) ** 2)).sum(0))
        rdv = dw[1 + d] - vd * dw[0]
        cs2 = g * p / rho
        tot = (B ** 2).sum(0) / rho + cs2
        cs = (0.5 * (tot - (tot ** 2 - 4 * cs2 * bd ** 2 / rho).clamp(min=0).sqrt())).clamp(min=0)
        cf = tot - cs
        af = ((cs2 - cs) / (cf - cs)).clamp(0, 1)
        As, af, cf, cs, sr = (1 - af).sqrt(), af.sqrt(), cf.sqrt(), cs.sqrt(), rho.sqrt()
        others = [(d + 1 + k) % nd for k in range(nd - 1)]
        if nd == 2:
            beta = [torch.where(B[others[0]] >= 0, 1.0, -1.0).to(B)]
        else:
            t = (B[others[0]] ** 2 + B[others[1]] ** 2).sqrt()
            h = torch.full_like(t, math.sqrt(0.5))
            beta = [torch.where(t > 1e-99, B[o] / t.clamp(min=1e-300), h) for o in others]
        bd = torch.where(bd.abs() < 1e-99, torch.full_like(bd, 1e-99), bd)
        sg = torch.copysign(torch.ones_like(bd), bd)
        bdv = sum(bt * dv[o] for bt, o in zip(beta, others)) * rho * sg
        bdb = sum(bt * db[o] for bt, o in zip(beta, others)) * cs2.sqrt() * sr
        bv = sum(bt * v[o] for bt, o in zip(beta, others)) * sg
        v2 = (v ** 2).sum(0)
        v2a2 = 0.5 * v2 + (2 - g) / (g - 1) * cs2
        half = 0.5 / cs2
        out = torch.zeros_like(dw)

        def fastslow(sign, c, w0, w1, c1, fast):
            # w0, c: the wave's own weight and speed; w1, c1: the other's
            s1 = -1.0 if fast else 1.0
            j = half * (w0 * (sign * c * rdv + dp) + w1 * (sign * s1 * c1 * bdv - s1 * bdb))
            q = (vd + sign * c).abs() * j
            out[0] += q * w0
            out[E] += q * (sign * s1 * w1 * c1 * bv + w0 * (v2a2 + c * (c + sign * vd)))
            out[1 + d] += q * w0 * (vd + sign * c)
            for bt, o in zip(beta, others):
                out[1 + o] += q * (w0 * v[o] + sign * s1 * w1 * c1 * bt * sg)
                out[E + 1 + o] += -s1 * q * w1 * cs2.sqrt() * bt / sr

        fastslow(1.0, cf, af, As, cs, True)
        fastslow(-1.0, cf, af, As, cs, True)
        fastslow(1.0, cs, As, af, cf, False)
        fastslow(-1.0, cs, As, af, cf, False)
        q = vd.abs() * (dw[0] - dp / cs2)  # entropy
        out[0] += q
        out[E] += q * 0.5 * v2
        out[1:1 + nd] += q * v
        q = vd.abs() * db[d]  # div B
        out[E] += q * bd
        out[E + 1 + d] += q
        if nd == 3:  # Alfven
            I, J = others
            av = (beta[1] * dv[I] - beta[0] * dv[J]) * 0.5 * rho
            ab = (beta[1] * db[I] - beta[0] * db[J]) * 0.5 * sr * sg
            cv = beta[1] * v[I] - beta[0] * v[J]
            for sign in (1.0, -1.0):
                q = (vd + sign * bd.abs() / sr).abs() * (sign * av - ab)
                out[E] += sign * q * cv
                out[1 + I] += sign * q * beta[1]
                out[1 + J] -= sign * q * beta[0]
                out[E + 1 + I] -= q * beta[1] * sg / sr
                out[E + 1 + J] += q * beta[0] * sg / sr
        return out, torch.maximum((vd + cf).abs().max(), (vd - cf).abs().max())

    def sweep(self, w, d, dt):
        ax, n, h = w.dim() - 1 - d, w.shape[w.dim() - 1 - d], self.dx[d]
        W = self.pad(w)
        line = self.cut(W, d, 0, n + 4)
        diff = line.narrow(ax, 1, n + 3) - line.narrow(ax, 0, n + 3)
        slope = self.limit(diff.narrow(ax, 1, n + 2), diff.narrow(ax, 0, n + 2))
        del diff
        s = 0.5 * slope.narrow(ax, 1, n)
        w1 = w - 0.5 * dt / h * (self.flux(w + s, d) - self.flux(w - s, d))
        w1 = self.powell(W, w, 0.5 * dt / self.nd, w1)
        W1 = self.pad(w1)
        c = self.cut(W1, d, 1, n + 2)
        L = c.narrow(ax, 0, n + 1) + 0.5 * slope.narrow(ax, 0, n + 1)
        R = c.narrow(ax, 1, n + 1) - 0.5 * slope.narrow(ax, 1, n + 1)
        F = 0.5 * (self.flux(L, d) + self.flux(R, d))
        if self.roe:
            q, cm = self.waves(L, R, d)
            F -= 0.5 * q
        else:
            c = self.cmax(0.5 * (L + R), d)
            F -= 0.5 * c * (R - L)
            cm = c.max()
        new = w - dt / h * (F.narrow(ax, 1, n) - F.narrow(ax, 0, n))
        return self.powell(W1, w1, dt / self.nd, new), cm / h

    def advance(self, w, steps, courant=0.8):
        rate = max(float(self.cmax(w, d).max()) / self.dx[d] for d in range(self.nd))
        rate, t = torch.tensor(rate, device=w.device, dtype=w.dtype), 0.0
        for it in range(steps):
            dt, rates = courant / rate, []
            order = range(self.nd) if it % 2 == 0 else range(self.nd - 1, -1, -1)
            for d in order:
                w, r = self.sweep(w, d, dt)
                rates.append(r)
            rate = torch.stack(rates).max()
            t = t + dt
        return w, float(t)


def exact(case, seed):
    c = dict(case)
    if c["job"] == "engine":
        _, w, dx, gamma = _state(c["physics"], _nx(c), c["init"], c["p0"], seed)
        w, t = _Scheme(c["physics"], dx, gamma, c["limiter"], c["bc"],
                       c["method"]).advance(w, c["steps"])
        return {"w": w.reshape(-1), "t": np.float64(t), "it": c["steps"]}
    specs = _batch_grids(c, seed) if c["job"] == "batch" else _server_grids(c, seed)
    ws, ts = [], []
    for physics, nx, init, steps, p0, sd in specs:
        _, w, dx, gamma = _state(physics, nx, init, p0, sd)
        lim = c.get("limiter", "minmod" if len(nx) == 2 else "woodward")
        w, t = _Scheme(physics, dx, gamma, lim, "cont" if c["job"] == "batch" else "periodic",
                       "tvdlf").advance(w, steps)
        ws.append(w.reshape(-1))
        ts.append(t)
    return {"w": torch.cat(ws), "t": torch.tensor(ts, dtype=torch.float64)}

