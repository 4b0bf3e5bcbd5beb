"""Performance cases of the hydro framework: the work that its users have it do.

A pass is what a host program does between two looks at its run: ``run(steps=...)`` on a uniform
grid (:class:`shaderous_b200.Sim`) or on the adaptive mesh (:class:`shaderous_b200.amr.AmrSim`),
with the totals where a report asks for them, or a set of requests given to the server and their
states taken back. A pass goes on from the state that the last one left, as a run does.

``exact`` is the scheme in float64 in plain torch: limited or parabolic edges, the density along
the adiabat, the Hancock half step, HLLC/HLL fluxes, the conservative update with the dual-energy
switch, and the CFL step. It covers uniform grids and served requests. The adaptive mesh has no such
value here: ghost filling, flux matching and re-meshing are the library's own subject.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from shaderous_b200 import Config, Problem, Sim, _abi
from shaderous_b200.amr import AmrConfig, AmrSim
from shaderous_b200.serve import Request, Server, ServerConfig

RHO_FLOOR, P_FLOOR, ETA_DUAL, SHOCK = 1e-10, 1e-12, 1e-3, 0.5
PERIODIC, OUTFLOW, REFLECT = 0, 1, 2
BC = {"periodic": PERIODIC, "outflow": OUTFLOW, "reflect": REFLECT}


# ---------------------------------------------------------------------------------------------
# The cases

def grid(name, n, problem, recon, steps, *, isentropic=True, riemann="hllc", bc="periodic", cfl=0.4, gamma=1.4,
         report=False):
    nx, ny, nz = n
    return {"name": name, "kind": "grid", "nx": nx, "ny": ny, "nz": nz, "problem": problem, "recon": recon,
            "isentropic": isentropic, "riemann": riemann, "bc": bc, "cfl": cfl, "gamma": gamma, "steps": steps,
            "report": report}


def mesh(name, ndim, nr, levels, cap, problem, radius, recon, steps, *, leaves, time_bins=0, bc="outflow", cfl=0.5,
         gamma=5 / 3):
    """`leaves`: blocks of the mesh at the start, for `work` (at least the roots, where it is not known)."""
    return {"name": name, "kind": "amr", "ndim": ndim, "nr": nr, "levels": levels, "cap": cap, "problem": problem,
            "radius": radius, "recon": recon, "steps": steps, "leaves": leaves, "time_bins": time_bins, "bc": bc,
            "cfl": cfl, "gamma": gamma}


def listed():
    return [
        # a shock tube, the smallest run there is: launches and the host's looks at the clock
        grid("sod_1d_512", (512, 1, 1), "sod", "minmod", 64, bc="outflow"),
        # the smallest 2D request of the served stream, run by itself
        grid("kh_2d_64", (64, 64, 1), "kh", "koren", 64),
        # an ordinary 2D run of odd sides, walls, the HLL solver, totals reported after it
        grid("blast_2d_301x219", (301, 219, 1), "blast", "vanleer", 32, isentropic=False, riemann="hll", bc="reflect",
             report=True),
        # the 2D configuration the benchmark states (1024^2, MC + HLLC)
        grid("kh_2d_1024", (1024, 1024, 1), "kh", "mc", 16, isentropic=False),
        # the reference's default scheme at its published 2D size
        grid("kh_2d_2048", (2048, 2048, 1), "kh", "koren", 8, cfl=0.8),
        # a small 3D run of odd sides with its totals
        grid("blast_3d_45x52x61", (45, 52, 61), "blast", "koren", 16, bc="outflow", cfl=0.5, report=True),
        # the reference's published 3D size, the default scheme
        grid("sedov_3d_256", (256, 256, 256), "sedov", "koren", 4, bc="outflow", cfl=0.8, gamma=5 / 3),
        # the headline: Taylor-Green, parabolic reconstruction
        grid("tgv_3d_512", (512, 512, 512), "tgv", "ppm", 1, gamma=5 / 3),
        # the adaptive Sedov blast as configured (levels 0-4), a young mesh
        mesh("sedov_amr_3d", 3, 8, 4, 2500, "sedov", 3.5, "koren", 32, leaves=736),
        # a grown blast: a hot rarefied bubble behind a refined shell, thousands of leaves
        mesh("bubble_amr_3d", 3, 8, 3, 12000, "bubble", 0.16, "koren", 32, leaves=6224),
        # the configured blast with per-block timesteps
        mesh("sedov_amr_3d_bins", 3, 8, 4, 2500, "sedov", 3.5, "koren", 64, leaves=736, time_bins=5),
        # requests of the served stream's kinds, small enough to share the block passes
        {"name": "serve_mixed", "kind": "serve", "requests": 6, "low2": 64, "high2": 320, "low3": 32, "high3": 64,
         "steps": 100, "recon": "koren", "isentropic": True, "pick": 11},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["1d", "2d", "2d", "3d", "3d", "amr2", "amr3", "serve"])
    recon = rng.choice(["minmod", "mc", "vanleer", "koren", "koren", "ppm"])
    common = {"isentropic": rng.random() < 0.7, "riemann": "hll" if rng.random() < 0.2 else "hllc",
              "bc": rng.choice(["periodic", "outflow", "reflect"]), "cfl": rng.choice([0.3, 0.4, 0.5, 0.8]),
              "gamma": rng.choice([1.4, 5 / 3]), "report": rng.random() < 0.3}
    bins = rng.choice([0, 0, 0, 4])
    if kind == "1d":
        c = grid("", (_log(rng, 48, 8192), 1, 1), rng.choice(["sod", "blast"]), recon, 64, **common)
    elif kind == "2d":
        n = (_log(rng, 40, 2200), _log(rng, 40, 2200), 1)
        c = grid("", n, rng.choice(["kh", "blast", "sod"]), recon, 8 if n[0] * n[1] > 1 << 20 else 32, **common)
    elif kind == "3d":
        n = [_log(rng, 24, 320) for _ in range(3)]
        c = grid("", n, rng.choice(["tgv", "blast", "sedov"]), recon, 4 if n[0] * n[1] * n[2] > 1 << 22 else 16, **common)
    elif kind == "amr2":
        nr, lev = rng.randint(3, 12), rng.randint(2, 4)
        c = mesh("", 2, nr, lev, 12000, "sedov" if bins else "bubble", 3.5 if bins else rng.uniform(0.08, 0.2),
                 rng.choice(["mc", "koren", "vanleer"]), 32, leaves=nr * nr, time_bins=bins,
                 bc=rng.choice(["periodic", "outflow", "reflect"]), cfl=rng.choice([0.3, 0.4, 0.5]))
    elif kind == "amr3":
        nr, lev = rng.randint(2, 6), rng.randint(2, 3)
        c = mesh("", 3, nr, lev, 7000, "sedov" if bins else "bubble", 3.5 if bins else rng.uniform(0.08, 0.16),
                 rng.choice(["mc", "koren", "minmod"]), 32, leaves=nr ** 3, time_bins=bins,
                 bc=rng.choice(["periodic", "outflow", "reflect"]), cfl=rng.choice([0.3, 0.4, 0.5]))
    else:
        c = {"kind": "serve", "requests": rng.randint(3, 8), "low2": 64, "high2": rng.choice([128, 240, 400]), "low3": 32,
             "high3": rng.choice([48, 64, 80]), "steps": 100, "recon": rng.choice(["mc", "koren"]),
             "isentropic": rng.random() < 0.7, "pick": rng.randrange(1 << 20)}
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------------------------
# Inputs

def _rand(seed, lo, hi, k):
    return float(np.random.default_rng([seed, k]).uniform(lo, hi))


def _config(c):
    b = BC[c["bc"]]
    n = (c["nx"], c["ny"], c["nz"])
    code = tuple(b if m > 1 else PERIODIC for m in n)
    dx = (2 * math.pi if c["problem"] == "tgv" else 1.0) / c["nx"]
    return Config(n=n, dx=dx, gamma=c["gamma"], bc_lo=code, bc_hi=code, cfl=c["cfl"], rho_floor=RHO_FLOOR, p_floor=P_FLOOR,
                  eta_dual=ETA_DUAL, shock_thresh=SHOCK, riemann=c["riemann"], recon=c["recon"], isentropic=c["isentropic"])


def _initial(c, seed):
    """The float32 conserved state (u1, u2) of a grid case, formed in float64 on the device and
    rounded once: (rho, momentum) and (E, e_int, rho s, 0) per cell, x fastest."""
    cfg = _config(c)
    n, dx, dev = cfg.n, cfg.dx, "cuda"
    ax = [((torch.arange(m, dtype=torch.float64, device=dev) + 0.5 - m / 2) * dx) for m in n]
    x, y, z = ax[0].view(1, 1, -1), ax[1].view(1, -1, 1), ax[2].view(-1, 1, 1)
    if n[1] == 1:
        y = y * 0
    if n[2] == 1:
        z = z * 0
    shape = (n[2], n[1], n[0])
    zero = torch.zeros((), dtype=torch.float64, device=dev)
    vx = vy = vz = s = zero
    rho = p = zero + 1
    r = lambda k, lo, hi: _rand(seed, lo, hi, k)  # noqa: E731
    either = lambda where, a, b: torch.where(where, zero + a, zero + b)  # noqa: E731
    kind = c["problem"]
    if kind == "sod":
        left = x < 0
        rho, p = either(left, r(0, 1, 10), 1.0), either(left, math.exp(r(1, 0, math.log(1000))), 1.0)
        s = left.double()
    elif kind == "kh":
        L = n[1] * dx
        inner = y.abs() < 0.25 * L
        g = torch.Generator(device=dev).manual_seed(seed)
        rho, vx, s = either(inner, r(0, 1.5, 2.5), 1.0), either(inner, 0.5, -0.5), inner.double()
        vy = 0.01 * torch.sin(4 * math.pi * (x / (n[0] * dx) + 0.5)) + 1e-3 * torch.randn(
            shape, dtype=torch.float64, device=dev, generator=g)
        p = zero + 2.5
    elif kind == "tgv":
        k = [2 * math.pi / (m * dx) for m in n]
        X, Y, Z = ((q + m * dx / 2) * kk for q, m, kk in zip((x, y, z), n, k))
        v = r(0, 0.8, 1.2)
        vx, vy = v * torch.sin(X) * torch.cos(Y) * torch.cos(Z), -v * torch.cos(X) * torch.sin(Y) * torch.cos(Z)
        p = zero + r(1, 90, 110)
    else:
        d2 = (x * x + y * y + z * z)
        radius = 3.5 * dx if kind == "sedov" else 0.15
        hot = d2.sqrt() < radius
        nd = 3 if n[2] > 1 else 2 if n[1] > 1 else 1
        if kind == "sedov":
            cells = max(1, int(hot.sum()))
            rho, p = zero + 1, either(hot, (c["gamma"] - 1) * r(0, 0.8, 1.2) / (cells * dx ** nd), 1e-5)
        else:
            rho, p = either(hot, r(0, 1, 10), 1.0), either(hot, math.exp(r(1, 0, math.log(1000))), 1.0)
        s = hot.double()
    e = p / (c["gamma"] - 1)
    u1 = torch.empty(shape + (4,), dtype=torch.float32, device=dev)
    u2 = torch.zeros(shape + (4,), dtype=torch.float32, device=dev)
    for i, v in enumerate((rho, rho * vx, rho * vy, rho * vz)):
        u1[..., i] = v
    u2[..., 0] = e + 0.5 * rho * (vx * vx + vy * vy + vz * vz)
    u2[..., 1] = e
    u2[..., 2] = rho * s
    return u1.view(-1, 4), u2.view(-1, 4)


class _Device:
    """A device array of the library as torch sees one; its owner lives as long as it is seen."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 3, "strides": None}


def _requests(c, seed):
    """The served requests: their sizes belong to the case, their parameters to the seed."""
    rng, par = np.random.default_rng(c["pick"]), np.random.default_rng(seed)
    out = []
    for i in range(c["requests"]):
        nd = 2 + i % 2
        lo, hi = (c["low2"], c["high2"]) if nd == 2 else (c["low3"], c["high3"])
        n = max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 16)) * 16)
        kind = ("kh", "blast", "sod")[i % 3]
        rr, pr = float(par.uniform(1, 10)), float(math.exp(par.uniform(0, math.log(1000))))
        if kind == "sod":
            p, bc = Problem("sod", a=(rr, 0, pr, 1, 0, 1), axis=0), OUTFLOW
        elif kind == "kh":
            p, bc = Problem("kh", a=(rr, 1, 0.5, 2.5, 0.01, 1e-3), seed=int(par.integers(1 << 62))), PERIODIC
        else:
            p, bc = Problem("blast", a=(rr, pr, 1, 1, 0.15)), OUTFLOW
        out.append(Request(ndim=nd, n=n, steps=c["steps"], problem=p, gamma=[1.4, 5 / 3][int(par.integers(2))], bc=bc))
    return out


def prepare(case, seed):
    c = case
    if c["kind"] == "grid":
        u1, u2 = _initial(c, seed)
        host = [torch.empty(u.shape, dtype=u.dtype, pin_memory=True) for u in (u1, u2)]
        for h, u in zip(host, (u1, u2)):
            h.copy_(u)
        sim = Sim(_config(c))
        sim.set_state(host[0].numpy(), host[1].numpy())
        sim.sync()
        return {"case": c, "sim": sim, "views": {}}
    if c["kind"] == "amr":
        b = (BC[c["bc"]],) * 3
        hyd = Config(gamma=c["gamma"], bc_lo=b, bc_hi=b, recon=c["recon"], isentropic=True, cfl=c["cfl"], p_floor=P_FLOOR)
        sim = AmrSim(AmrConfig(hydro=hyd, ndim=c["ndim"], nr=c["nr"], max_level=c["levels"], cap=c["cap"], refine_hi=0.1,
                               refine_lo=0.05, regrid_every=8, time_bins=c["time_bins"],
                               time_bins_always=c["time_bins"] > 0))
        if c["problem"] == "sedov":
            sim.reset(Problem("sedov", a=(1.0, 1e-5, _rand(seed, 0.8, 1.2, 0), c["radius"])))
        else:
            # the inside of a blast: hot and thin against what lies ahead of it
            sim.reset(Problem("blast", a=(_rand(seed, 0.008, 0.012, 0), _rand(seed, 20, 40, 1), 1.0, 0.01, c["radius"])))
        return {"case": c, "sim": sim, "pinned": None}
    hyd = Config(recon=c["recon"], isentropic=c["isentropic"], cfl=0.4, p_floor=P_FLOOR)
    return {"case": c, "server": Server(ServerConfig(hydro=hyd, budget_bytes=4e9, keep_states=True)),
            "requests": _requests(c, seed)}


# ---------------------------------------------------------------------------------------------
# A pass

def _totals(d):
    return np.array([d.mass, *d.momentum, d.e_kin, d.e_int, d.e_tot, d.max_mach])


def run(state):
    c = state["case"]
    if c["kind"] == "grid":
        sim, views = state["sim"], state["views"]
        r = sim.run(steps=c["steps"])
        out = {"t": r.t, "dt": r.dt}
        if c["report"]:
            out["totals"] = _totals(sim.diagnostics())
        for name, ptr in zip(("u1", "u2"), sim.state_device()):
            if ptr not in views:  # (two parities a buffer)
                views[ptr] = torch.as_tensor(_Device(ptr, (sim.ncell, 4), sim), device="cuda")
            out[name] = views[ptr]
        return out
    if c["kind"] == "amr":
        sim = state["sim"]
        r = sim.run(steps=c["steps"])
        _, levels, coords = sim.leaves()
        # the leaves' state through the C interface into the caller's own pinned memory, kept and grown
        want = len(levels) * 16 ** c["ndim"]
        if state["pinned"] is None or state["pinned"][0].shape[0] < want:
            state["pinned"] = [torch.empty((want + want // 4, 4), dtype=torch.float32, pin_memory=True) for _ in range(2)]
        u1, u2 = state["pinned"]
        rc = _abi.load().shz_amr_get_leaves_state(sim._h, C.c_void_p(u1.data_ptr()), C.c_void_p(u2.data_ptr()))
        if rc:
            raise RuntimeError("shz_amr_get_leaves_state: %d" % rc)
        return {"t": r.t, "dt": r.dt, "levels": levels, "coords": coords, "u1": u1[:want], "u2": u2[:want]}
    server, reqs = state["server"], state["requests"]
    ids = [server.submit(q) for q in reqs]
    server.drain()
    return [{"t": server.result(i).t, "state": list(server.state(i, q))} for i, q in zip(ids, reqs)]


# ---------------------------------------------------------------------------------------------
# The work

# Floating-point operations a cell and axis cannot do without, counted from the scheme's formulas: the
# edges of six primitives (and the density along the adiabat), a half step, two face states and a flux.
EDGES = {"minmod": 50, "mc": 70, "vanleer": 60, "koren": 150, "ppm": 200}


def work(case):
    c = case
    per = lambda nd, isen: nd * (EDGES[c["recon"]] + (60 if isen and c["recon"] != "ppm" else 0) + 160) + 60  # noqa: E731
    if c["kind"] == "grid":
        cells = c["nx"] * c["ny"] * c["nz"]
        nd = 3 if c["nz"] > 1 else 2 if c["ny"] > 1 else 1
        # a state that the chip's own memory holds (126 MB of L2) need cross HBM once a pass; a larger one each step
        trips = 1 if 32 * cells <= 100e6 else c["steps"]
        return {"bytes": 64.0 * cells * trips, "flops": float(cells * c["steps"] * per(nd, c["isentropic"]))}
    if c["kind"] == "amr":
        cells = c["leaves"] * 16 ** c["ndim"]
        # with per-block timesteps most blocks take a few of a cycle's substeps: a quarter, as a bound from below
        share = 0.25 if c["time_bins"] else 1.0
        trips = 1 if 32 * cells <= 100e6 else c["steps"] * share
        return {"bytes": 64.0 * cells * trips + 32.0 * cells, "flops": float(cells * c["steps"] * share * per(c["ndim"], True))}
    cells = [(q.ndim, q.cells) for q in _requests(c, 0)]
    return {"bytes": 64.0 * sum(n for _, n in cells), "flops": float(sum(n * per(d, c["isentropic"]) for d, n in cells) * c["steps"])}


def tolerance(case):
    # float32 state against float64 after a pass: 3e-8 to 7e-7 (a few roundings a step, and what a
    # shear layer or a shock makes of them); four times that. The adaptive mesh takes more steps a
    # pass and restricts and prolongs in between.
    return {"rel": 1e-5, "max": 1e-3} if case["kind"] == "amr" else {"rel": 3e-6, "max": 3e-4}


# ---------------------------------------------------------------------------------------------
# The scheme in float64

def _limit(kind, a, b, scale):
    same = a * b > 0
    zero = torch.zeros_like(a)
    if kind == "minmod":
        return torch.where(same, torch.sign(a) * torch.minimum(a.abs(), b.abs()), zero)
    if kind == "mc":
        return torch.where(same, torch.sign(a) * torch.minimum(2 * torch.minimum(a.abs(), b.abs()), 0.5 * (a + b).abs()), zero)
    if kind == "vanleer":
        return torch.where(same, 2 * a * b / torch.where(same, a + b, 1.0), zero)
    free = (a + 2 * b) / 3
    lim = torch.where(same, torch.sign(b) * torch.minimum(2 * torch.minimum(a.abs(), b.abs()), free.abs()), zero)
    s2 = (0.01 * scale) ** 2 if torch.is_tensor(scale) else zero
    w = (1.5 - (a * a + b * b) / s2.clamp_min(1e-30)).clamp(0, 1)
    return lim + (free - lim) * w


def _slope(dl, dr):
    d = 0.5 * (dl + dr)
    return torch.where(dl * dr > 0, torch.sign(d) * torch.minimum(d.abs(), 2 * torch.minimum(dl.abs(), dr.abs())), torch.zeros_like(d))


def _ppm(m2, m, a, p, p2):
    d0 = _slope(a - m, p - a)
    al = 0.5 * (m + a) - (d0 - _slope(m - m2, a - m)) / 6
    ar = 0.5 * (a + p) - (_slope(p - a, p2 - p) - d0) / 6
    flat = (ar - a) * (a - al) <= 0
    da, a6 = ar - al, 6 * (a - 0.5 * (al + ar))
    low = da * a6 > da * da
    high = ~low & (-da * da > da * a6)
    lo = torch.where(flat, a, torch.where(low, 3 * a - 2 * ar, al))
    hi = torch.where(flat, a, torch.where(high, 3 * a - 2 * al, ar))
    return 2 * (hi - a), 2 * (a - lo)


class _Exact:
    def __init__(self, n, dx, gamma, bc, cfl, recon, isentropic, hll, u1, u2):
        self.n, self.dx, self.gamma, self.bc, self.cfl = n, dx, gamma, bc, cfl
        self.recon, self.isen, self.hll = recon, isentropic and recon != "ppm", hll
        self.nd = 3 if n[2] > 1 else 2 if n[1] > 1 else 1
        shape = (n[2], n[1], n[0])
        self.U = [u.double().reshape(shape) for u in (u1[:, 0], u1[:, 1], u1[:, 2], u1[:, 3], u2[:, 0], u2[:, 1], u2[:, 2])]
        self.t = self.dt = 0.0

    def pad(self, x, axis, k, sign=1.0):
        """x with k ghosts at both ends of an axis, through the boundary; sign: what a wall does to it."""
        n, dim = self.n[axis], 2 - axis
        i = torch.arange(-k, n + k, device=x.device)
        if self.bc == PERIODIC:
            return x.index_select(dim, i % n)
        if self.bc == OUTFLOW:
            return x.index_select(dim, i.clamp(0, n - 1))
        out = (i < 0) | (i >= n)
        j = torch.where(i < 0, -1 - i, torch.where(i >= n, 2 * n - 1 - i, i)).clamp(0, n - 1)
        y = x.index_select(dim, j)
        if sign < 0:
            y = y * torch.where(out, -1.0, 1.0).to(x.dtype).view([-1 if d == dim else 1 for d in range(3)])
        return y

    def prims(self):
        U = self.U
        rho = U[0].clamp_min(RHO_FLOOR)
        return [rho, U[1] / rho, U[2] / rho, U[3] / rho, ((self.gamma - 1) * U[5]).clamp_min(P_FLOOR), U[6] / rho]

    def edges(self, W, axis):
        """Edge increments (upper, lower) of the cells -1 .. n along an axis."""
        n, dim = self.n[axis], 2 - axis
        k = 3 if self.recon == "ppm" else 2
        P = [self.pad(w, axis, k, -1.0 if v == 1 + axis else 1.0) for v, w in enumerate(W)]
        at = lambda x, o: x.narrow(dim, k - 1 + o, n + 2)  # noqa: E731
        if self.recon == "ppm":
            both = [_ppm(*(at(x, o) for o in (-2, -1, 0, 1, 2))) for x in P]
            return [b[0] for b in both], [b[1] for b in both]
        m, c, p = ([at(x, o) for x in P] for o in (-1, 0, 1))
        cs = (self.gamma * c[4] / c[0]).sqrt()
        scale = [c[0], cs, cs, cs, c[4], None]
        su = [_limit(self.recon, c[v] - m[v], p[v] - c[v], scale[v]) for v in range(6)]
        sd = [_limit(self.recon, p[v] - c[v], c[v] - m[v], scale[v]) for v in range(6)]
        if self.isen:
            gi = 1 / self.gamma
            tl, tr = m[0] * (c[4] / m[4]) ** gi - c[0], p[0] * (c[4] / p[4]) ** gi - c[0]
            fade = lambda x: (2 - x).clamp(0, 1)  # noqa: E731
            dv = lambda a, b: ((a[1] - b[1]) ** 2 + (a[2] - b[2]) ** 2 + (a[3] - b[3]) ** 2).sqrt()  # noqa: E731
            room = (fade(torch.maximum((m[4] - c[4]).abs(), (p[4] - c[4]).abs()) / (0.2 * c[4]))
                    * fade(torch.maximum(tl.abs(), tr.abs()) / (0.01 * c[0]))
                    * fade(torch.maximum(dv(p, c), dv(c, m)) / (0.1 * cs.clamp_min(1e-30))))
            bound = torch.maximum(0.25 * torch.minimum((c[0] - m[0]).abs(), (p[0] - c[0]).abs()), 0.01 * c[0] * room)
            for s, far, near, nb, inc in ((1, -tl, tr, p, su), (-1, tr, -tl, m, sd)):
                pf = (c[4] + 0.5 * s * inc[4]).clamp_min(1e-30)
                rf = (c[0] + 0.5 * s * _limit(self.recon, far, near, c[0])) * (pf / c[4]) ** gi
                rf = torch.minimum(torch.maximum(rf, torch.minimum(c[0], nb[0])), torch.maximum(c[0], nb[0]))
                inc[0] = inc[0] + torch.minimum(torch.maximum(2 * s * (rf - c[0]) - inc[0], -bound), bound)
        return su, sd

    def flux(self, L, R, axis, w):
        g = self.gamma
        order = [1 + axis, 1 + (axis + 1) % 3, 1 + (axis + 2) % 3]
        sides = []
        for q in (L, R):
            rho, p = q[0].clamp_min(RHO_FLOOR), q[4].clamp_min(P_FLOOR)
            v = [q[k] for k in order]
            ei = p / (g - 1)
            e = ei + 0.5 * rho * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
            sides.append((rho, v, p, (g * p / rho).sqrt(), e, ei, q[5]))
        (rl, vl, pl, cl, el, eil, s_l), (rr, vr, pr, cr, er, eir, s_r) = sides
        sl, sr = torch.minimum(vl[0] - cl, vr[0] - cr), torch.maximum(vl[0] + cl, vr[0] + cr)
        ql, qr = rl * (sl - vl[0]), rr * (sr - vr[0])
        sm = (pr - pl + vl[0] * ql - vr[0] * qr) / (ql - qr)
        Ul, Ur = [rl] + [rl * v for v in vl] + [el], [rr] + [rr * v for v in vr] + [er]
        Fl = [Ul[1], Ul[1] * vl[0] + pl, Ul[2] * vl[0], Ul[3] * vl[0], (el + pl) * vl[0]]
        Fr = [Ur[1], Ur[1] * vr[0] + pr, Ur[2] * vr[0], Ur[3] * vr[0], (er + pr) * vr[0]]
        left = sm >= 0
        pick = lambda a, b: torch.where(left, a, b)  # noqa: E731
        sk, qk, rk, pk, ek = pick(sl, sr), pick(ql, qr), pick(rl, rr), pick(pl, pr), pick(el, er)
        vk = [pick(a, b) for a, b in zip(vl, vr)]
        f = qk / (sk - sm)
        star = [f, f * sm, f * vk[1], f * vk[2], f * (ek / rk + (sm - vk[0]) * (sm + pk / qk))]
        F = []
        for i in range(5):
            h = (sr * Fl[i] - sl * Fr[i] + sl * sr * (Ur[i] - Ul[i])) / (sr - sl)
            k = pick(Fl[i], Fr[i]) + sk * (star[i] - pick(Ul[i], Ur[i]))
            k = h if self.hll else k + (h - k) * w
            F.append(torch.where(sl >= 0, Fl[i], torch.where(sr <= 0, Fr[i], k)))
        vn = torch.where(sl >= 0, vl[0], torch.where(sr <= 0, vr[0], sm))
        up = F[0] >= 0
        out = [F[0], None, None, None, F[4], F[0] * torch.where(up, eil / rl, eir / rr), F[0] * torch.where(up, s_l, s_r), vn]
        for i, k in enumerate(order):
            out[k] = F[1 + i]
        return out

    def step(self):
        W = self.prims()
        cs = (self.gamma * W[4] / W[0]).sqrt()
        rate = float((W[1].abs() + W[2].abs() + W[3].abs() + 3 * cs).max())
        self.dt = self.cfl * self.dx / rate
        self.t += self.dt
        h, axes = 0.5 * self.dt / self.dx, range(self.nd)
        inc = [self.edges(W, a) for a in axes]
        own = [[[x.narrow(2 - a, 1, self.n[a]) for x in s] for s in inc[a]] for a in axes]
        adv = [sum(W[1 + a] * 0.5 * (own[a][0][v] + own[a][1][v]) for a in axes) for v in range(6)]
        div = sum(0.5 * (own[a][0][1 + a] + own[a][1][1 + a]) for a in axes)
        q = [w - h * d for w, d in zip(W, adv)]
        q[0] = q[0] - h * W[0] * div
        q[4] = q[4] - h * W[0] * cs * cs * div
        for a in axes:
            q[1 + a] = q[1 + a] - h * 0.5 * (own[a][0][4] + own[a][1][4]) / W[0]
        fall, big, conv, jump = 0.0, 0.0, 0.0, None
        for a in axes:
            su, sd = own[a]
            fall = torch.minimum(torch.minimum(0.5 * su[0], -0.5 * sd[0]), torch.as_tensor(fall, dtype=torch.float64, device=su[0].device))
            big = torch.maximum(torch.maximum(su[4].abs(), sd[4].abs()), torch.as_tensor(big, dtype=torch.float64, device=su[0].device))
            v, p = self.pad(W[1 + a], a, 1, -1.0), self.pad(W[4], a, 1)
            m_, p_ = ((x.narrow(2 - a, 0, self.n[a]), x.narrow(2 - a, 2, self.n[a])) for x in (v, p))
            conv = conv + m_[1] - m_[0]
            j = (p_[1] - p_[0]).abs() > SHOCK * torch.minimum(p_[0], p_[1])
            jump = j if jump is None else jump | j
        flag = ((conv < 0) & jump).double()
        first = ~((q[0] + fall > 0) & (q[4] - 0.5 * big > 0))
        q = [torch.where(first, w, x) for w, x in zip(W, q)]
        keep = (~first).double()
        del own, adv
        acc = [torch.zeros_like(W[0]) for _ in range(8)]
        for a in axes:
            n, dim = self.n[a], 2 - a
            lo, hi = (lambda x: x.narrow(dim, 0, n + 1)), (lambda x: x.narrow(dim, 1, n + 1))
            e = [self.pad(x, a, 1, -1.0 if v == 1 + a else 1.0) for v, x in enumerate(q)]
            k, f = self.pad(keep, a, 1), self.pad(flag, a, 1)
            L = [lo(x) + 0.5 * lo(k) * lo(s) for x, s in zip(e, inc[a][0])]
            R = [hi(x) - 0.5 * hi(k) * hi(s) for x, s in zip(e, inc[a][1])]
            inc[a] = None
            F = self.flux(L, R, a, torch.maximum(lo(f), hi(f)))
            for v in range(8):
                acc[v] += F[v].narrow(dim, 0, n) - F[v].narrow(dim, 1, n)
            del L, R, F, e
        U, r = self.U, self.dt / self.dx
        rho = (U[0] + r * acc[0]).clamp_min(RHO_FLOOR)
        mom = [U[1 + i] + r * acc[1 + i] for i in range(3)]
        E = U[4] + r * acc[4]
        eint = U[5] + r * (acc[5] + q[4].clamp_min(P_FLOOR) * acc[7])
        ke = 0.5 * (mom[0] ** 2 + mom[1] ** 2 + mom[2] ** 2) / rho
        low = P_FLOOR / (self.gamma - 1)
        total = (E - ke > ETA_DUAL * E) & (E - ke >= low)
        own_e = eint.clamp_min(low)
        self.U = [rho, *mom, torch.where(total, E, ke + own_e), torch.where(total, E - ke, own_e), U[6] + r * acc[6]]

    def state(self):
        U = self.U
        return [torch.stack([x.reshape(-1) for x in part], dim=1) for part in (U[:4], (U[4], U[5], U[6], torch.zeros_like(U[0])))]

    def totals(self):
        U, dv = self.U, self.dx ** self.nd
        rho = U[0].clamp_min(RHO_FLOOR)
        v2 = (U[1] ** 2 + U[2] ** 2 + U[3] ** 2) / rho ** 2
        ke = 0.5 * rho * v2
        cs = (self.gamma * ((self.gamma - 1) * U[5]).clamp_min(P_FLOOR) / rho).sqrt()
        sums = [rho, U[1], U[2], U[3], ke, U[4] - ke, U[4]]
        return np.array([float(x.sum()) * dv for x in sums] + [float((v2.sqrt() / cs).max())])


def _served_state(req):
    """A request's initial state: the library's built-in problems at cell centres, in float64, rounded once."""
    n, nd, a, kind = req.n, req.ndim, req.problem.a, req.problem.kind
    x = (np.arange(n) + 0.5 - n / 2.0) / n
    z = x if nd == 3 else np.zeros(1)
    X, Y, Z = x[None, None, :], x[None, :, None], z[:, None, None]
    shape = (len(z), n, n)
    one = np.ones(shape)
    vx, vy = 0 * one, 0 * one
    if kind == "kh":
        cell = np.arange(one.size, dtype=np.uint64).reshape(shape)

        def mix(v):  # SplitMix64
            v = v + np.uint64(0x9E3779B97F4A7C15)
            v = (v ^ (v >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
            v = (v ^ (v >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
            return v ^ (v >> np.uint64(31))

        unit = lambda v: ((v >> np.uint64(11)).astype(np.float64) + 0.5) / 9007199254740992.0  # noqa: E731
        s64 = np.uint64(req.problem.seed)
        g = np.sqrt(-2 * np.log(unit(mix(s64 ^ (cell * np.uint64(2)))))) * np.cos(
            2 * math.pi * unit(mix(s64 ^ (cell * np.uint64(2) + np.uint64(1)))))
        inner = (np.abs(Y) < 0.25) & (one > 0)
        rho, vx, p = np.where(inner, a[0], a[1]), np.where(inner, a[2], -a[2]), a[3] * one
        vy = a[4] * np.sin(4 * math.pi * (X + 0.5)) + a[5] * g
    elif kind == "sod":
        inner = (X < 0) & (one > 0)
        rho, p = np.where(inner, a[0], a[3]), np.where(inner, a[2], a[5])
    else:
        inner = (np.sqrt(X * X + Y * Y + Z * Z) < a[4]) & (one > 0)
        rho, p = np.where(inner, a[0], a[2]), np.where(inner, a[1], a[3])
    e = p / (req.gamma - 1)
    u1 = np.stack([rho, rho * vx, rho * vy, 0 * one], -1).reshape(-1, 4).astype(np.float32)
    u2 = np.stack([e + 0.5 * rho * (vx * vx + vy * vy), e, rho * inner, 0 * one], -1).reshape(-1, 4).astype(np.float32)
    return torch.from_numpy(u1).cuda(), torch.from_numpy(u2).cuda()


def exact(case, seed):
    c = case
    if c["kind"] == "amr":
        return None
    if c["kind"] == "grid":
        cfg = _config(c)
        x = _Exact(cfg.n, cfg.dx, c["gamma"], BC[c["bc"]], c["cfl"], c["recon"], c["isentropic"], c["riemann"] == "hll",
                   *_initial(c, seed))
        for _ in range(c["steps"]):
            x.step()
        u1, u2 = x.state()
        out = {"t": x.t, "dt": x.dt, "u1": u1, "u2": u2}
        if c["report"]:
            out["totals"] = x.totals()
        return out
    out = []
    for q in _requests(c, seed):
        n = (q.n, q.n, q.n if q.ndim == 3 else 1)
        x = _Exact(n, 1.0 / q.n, q.gamma, q.bc, 0.4, c["recon"], c["isentropic"], False, *_served_state(q))
        for _ in range(q.steps):
            x.step()
        out.append({"t": x.t, "state": [u.cpu() for u in x.state()]})
    return out
