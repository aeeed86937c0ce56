"""Workloads of the SPH engine, each one pass through its public entry points.

kind "update"  SmoothParticleSystem.run(dt, steps) on numpy arrays: the
               reference's own API, in its own arithmetic (fp64) by default
kind "steps"   one simulation of an Engine on CUDA tensors: set_state, advance,
               get_state and properties -- a run between two snapshots
kind "batch"   many simulations in one Engine: set_state of each, one advance,
               get_state of each, as the job server drives its engines
kind "eval"    Engine.derivatives at a given state, for a caller with an
               integrator of its own
kind "pairs"   VerletList.build: the exported pair list with its geometry
kind "splat"   interpolate.splash_map_2d / splash_map_3d

A fluid is a lattice of nx x ny (x nz) particles at number density `density`
with 10% jitter and Maxwell velocities; its smoothing lengths are given in
units of the lattice spacing of the 2D and 3D fluids of the repository's
benchmark (supports of 3 and 6 spacings in 2D; 2.735 and 5.148 at n = 0.7 in
3D, about 60 and 400 neighbours).

A mixed-precision engine computes densities, rates and the changes of v and u
in FP32 and positions in FP64; `run` returns each in the type in which it was
computed.
"""
import math

import numpy as np
import torch

from pyticles_gb300 import Engine, interpolate
from pyticles_gb300._abi import make_params
from pyticles_gb300.box import PeriodicBox
from pyticles_gb300.forces import SpamComplete
from pyticles_gb300.neighbour_list import VerletList
from pyticles_gb300.particles import SmoothParticleSystem

A, B, KB = 2.0, 0.5, 1.0     # van der Waals a, b, k_B (the package's defaults)
TEMP = 0.6
DT = 1e-3
ALPHA, BETA, EPS = 1.0, 0.1, 0.01   # viscosity, the package's defaults
STAGES = {"euler": 1, "ieuler": 2, "rk4": 4}


# ---- the cases -------------------------------------------------------------

def fluid(**kw):
    c = {"kind": "steps", "dim": 2, "nx": 32, "ny": 32, "nz": 1, "density": 1.0, "sims": 1,
         "kernel": "lucy", "viscosity": True, "heat": False, "integrator": "ieuler",
         "precision": "mixed", "scheme": 0, "thermostat": False, "steps": 1}
    c.update(kw)
    return c


def fluid3d(side, **kw):
    kw = {"kernel": "cubic", "heat": True, "density": 0.7, **kw}
    return fluid(dim=3, nx=side, ny=side, nz=side, **kw)


def listed():
    return [
        # the smallest use: a script that calls update(dt) on the plain small
        # configuration (32 x 32, fp64) and reads the arrays after each step
        fluid(name="update 2d 1k fp64", kind="update", precision="fp64"),
        # the reference is written for 3D: a small 3D system, run(dt, 4)
        fluid3d(13, name="update 3d 2k fp64", kind="update", precision="fp64", kernel="lucy",
                heat=False, steps=4),
        # the smallest job of the served workload on an engine with its
        # default knobs: launches and latency count
        fluid(name="run 2d 1k", steps=20),
        # a served 2D job of ordinary size on cell windows (the server's 2D
        # default), rectangular and odd
        fluid(name="run 2d 200k windows", nx=449, ny=443, steps=8),
        # the benchmark's fluid on the knobs that its tuner picks
        fluid(name="run 2d 1M lists", nx=1024, ny=1024, scheme=2, steps=16),
        # the plain fp64 arm on an ordinary size
        fluid(name="run 2d 65k fp64", nx=255, ny=257, precision="fp64", steps=2),
        # a served 3D job on cluster pairs (the server's 3D default)
        fluid3d(47, name="run 3d 104k clusters", scheme=1, steps=8),
        # the benchmark's 3D fluid on the knobs that its tuner picks
        fluid3d(128, name="run 3d 2M lists", scheme=2, steps=3),
        # independent thermostatted simulations of mixed sizes in one engine
        fluid(name="batch 2d 24 sims lists", kind="batch", nx=256, ny=256, sims=24,
              density=0.65, scheme=2, thermostat=True, steps=16),
        # rates alone, for a caller's own integrator: the Debrun kernel in 3D
        fluid3d(59, name="eval 3d 205k debrun", kind="eval", kernel="debrun", heat=False),
        # the neighbour list as data: pairs, separations, relative velocities
        fluid(name="pairs 2d 16k", kind="pairs", nx=126, ny=127, precision="fp64"),
        # a density picture of a simulation's particles
        fluid(name="splat 2d 100k", kind="splat", nx=317, ny=316, precision="fp64"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _sides(rng, dim, n):
    """Sides of a lattice of about n particles, rectangular and odd."""
    s = n ** (1.0 / dim)
    f = rng.uniform(0.9, 1.1)
    nx, ny = max(10, round(s * f)), max(10, round(s / f))
    nz = max(10, round(n / (nx * ny))) if dim == 3 else 1
    return {"nx": nx, "ny": ny, "nz": nz}


def draw(rng):
    kind = rng.choices(["steps", "update", "batch", "eval", "pairs", "splat"],
                       [9, 3, 2, 2, 1, 1])[0]
    dim = 3 if rng.random() < 0.4 else 2
    c = fluid(kind=kind, dim=dim)
    c["precision"] = "fp64" if kind in ("pairs", "splat") or (
        kind != "batch" and rng.random() < (0.75 if kind == "update" else 0.2)) else "mixed"
    fp64 = c["precision"] == "fp64"
    top = {"steps": 3e5 if fp64 else 9e5, "update": 2e4, "batch": 1e5, "eval": 5e5,
           "pairs": 3e4, "splat": 3e5}[kind]
    if fp64 and kind == "eval":
        top = 2e5
    if dim == 3:
        top *= 0.5
    c.update(_sides(rng, dim, _log(rng, 900 if dim == 2 else 1500, top)))
    c["density"] = round(rng.uniform(0.55, 0.75), 3) if dim == 3 else rng.choice(
        [1.0, round(rng.uniform(0.4, 0.9), 3)])
    # the kernels and options by how often they are used
    c["kernel"] = (rng.choices(["lucy", "cubic", "gaussian"], [6, 1, 1]) if dim == 2 else
                   rng.choices(["cubic", "lucy", "debrun"], [4, 2, 1]))[0]
    c["viscosity"] = rng.random() < 0.8
    c["heat"] = rng.random() < (0.7 if dim == 3 else 0.15)
    if kind in ("steps", "update"):
        c["integrator"] = rng.choices(["ieuler", "rk4", "euler"], [6, 1, 1])[0]
    if c["precision"] == "mixed":
        c["scheme"] = rng.choice([0, 2, 1] if dim == 3 else [0, 2])
    if kind in ("steps", "update", "batch"):
        n = c["nx"] * c["ny"] * c["nz"]
        cost = n * (400 if dim == 3 else 113) * STAGES[c["integrator"]] * (20 if fp64 else 1)
        c["steps"] = max(1, min(20, int(rng.uniform(0.2, 1.0) * 2.4e9 / cost)))
    if kind == "batch":
        c["sims"] = rng.randint(3, 32)
        c["thermostat"] = rng.random() < 0.7
        c["steps"] = min(c["steps"], 12)
        if dim == 3:
            c["sims"] = min(c["sims"], 10)
    return c


# ---- inputs ----------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _lengths(case):
    """(h_short, h_long, cutoff) of the case's fluid."""
    if case["dim"] == 2:
        s = case["density"] ** -0.5
        short, long_ = 3.0 * s, 6.0 * s
    else:
        s = (0.7 / case["density"]) ** (1.0 / 3.0)
        short, long_ = 2.735 * s, 5.148 * s
    if case["kernel"] == "cubic":              # support 2 h
        return short / 2, long_ / 2, long_
    if case["kernel"] == "gaussian":           # cut off at 3 h of the long length
        return long_ / 6, long_ / 3, long_
    return short, long_, long_


def _sim_sides(case):
    """Lattice sides of each simulation: in a batch the sizes run from 1/8 of
    the largest side up to it, evenly in their logarithm."""
    sides = [case["nx"], case["ny"], case["nz"]][:case["dim"]]
    k = case["sims"]
    if k == 1:
        return [sides]
    return [[max(10, round(s * 8.0 ** (j / (k - 1) - 1.0))) for s in sides] for j in range(k)]


def _system(case, sides, seed):
    """box, r, v, m, u of one simulation (float64, on the GPU)."""
    dim, dev = case["dim"], _device()
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    s = case["density"] ** (-1.0 / dim)
    axes = [(torch.arange(k, device=dev, dtype=torch.float64) + 0.5) * s for k in sides]
    r = torch.stack([x.reshape(-1) for x in torch.meshgrid(*axes, indexing="ij")], dim=1)
    r += 0.1 * s * (2.0 * torch.rand(r.shape, generator=g, device=dev, dtype=torch.float64) - 1.0)
    v = math.sqrt(TEMP) * torch.randn(r.shape, generator=g, device=dev, dtype=torch.float64)
    v -= v.mean(dim=0, keepdim=True)
    m = torch.ones(len(r), device=dev, dtype=torch.float64)
    # u = k_B T - a rho at the mean density, with a spread as a field that has
    # been running for a while
    u = torch.full((len(r),), KB * TEMP - A * case["density"], device=dev, dtype=torch.float64)
    u += 0.02 * torch.randn(len(r), generator=g, device=dev, dtype=torch.float64)
    return [k * s for k in sides], r.contiguous(), v.contiguous(), m, u


def _systems(case, seed):
    return [_system(case, sides, 1000 * seed + k) for k, sides in enumerate(_sim_sides(case))]


def _params(case, box):
    hs, hl, cut = _lengths(case)
    return make_params(dim=case["dim"], kernel=case["kernel"], box=box, h_short=hs, h_long=hl,
                       cutoff=cut, viscosity=case["viscosity"], heat_flux=case["heat"], dt=DT,
                       integrator=case["integrator"], thermostat=case["thermostat"],
                       thermostat_temp=TEMP)


def _host_system(case, seed):
    box, r, v, m, u = _systems(case, seed)[0]
    hs, hl, cut = _lengths(case)
    ext = list(box) + [1.0] * (3 - case["dim"])
    n = len(r)
    p = SmoothParticleSystem(n, d=case["dim"], maxn=n, hshort=hs, hlong=hl,
                             simbox=PeriodicBox(xmax=ext[0], ymax=ext[1], zmax=ext[2]),
                             integrator=case["integrator"], precision=case["precision"],
                             pair_scheme=case["scheme"])
    start = [x.cpu().numpy() for x in (r, v, m, u)]
    p.r[:], p.v[:], p.m[:], p.u[:] = start
    return p, start, cut


SKIN = 1.0   # the exported list's tolerance (the class's default), in quadrature


def _numbered(case, seed):
    """r, v for the pair list: one set of positions for every seed, so that the
    list has one length, with the particles numbered in an order of the seed's
    (a run leaves them in no order) and velocities of the seed's."""
    r = _systems(case, 1)[0][1]
    _, other, v, _, _ = _systems(case, seed)[0]
    return r[torch.argsort(other[:, 0].frac())].contiguous(), v


def _grid(case, box):
    """The picture's pixels: about two to a lattice spacing, at most 768."""
    k = [min(768, 2 * s + 1) for s in (case["nx"], case["ny"])]
    return [np.arange(k[a]) * (box[a] / k[a]) for a in (0, 1)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "update":
        p, start, cut = _host_system(case, seed)
        nl = VerletList(p, cutoff=cut, tolerance=0.0)
        p.nlists.append(nl)
        p.nl_default = nl
        on = 1.0 if case["viscosity"] else 0.0
        p.forces.append(SpamComplete(p, nl, cgrad=0.0, eta=ALPHA * on, zeta=BETA * on,
                                     kernel=case["kernel"], heat_flux=case["heat"]))
        return {"case": case, "p": p, "start": start}
    if kind == "pairs":
        p, _, cut = _host_system(case, seed)
        r, v = _numbered(case, seed)
        p.r[:], p.v[:] = r.cpu().numpy(), v.cpu().numpy()
        return {"case": case, "nl": VerletList(p, cutoff=cut, tolerance=SKIN)}
    if kind == "splat":
        box, r, v, m, u = _systems(case, seed)[0]
        n = len(r)
        rho = case["density"] * (1.0 + 0.05 * (u - u.mean()))
        hs = _lengths({**case, "kernel": "lucy"})[0]
        x, y = _grid(case, box)
        return {"case": case, "x": x, "y": y, "z": 0.5 * box[-1], "r": r.cpu().numpy(),
                "m": m.cpu().numpy(), "rho": rho.cpu().numpy(), "a": u.cpu().numpy(),
                "h": np.full(n, hs), "bounds": (0.0, box[0], 0.0, box[1]), "cutoff": hs}
    systems = _systems(case, seed)
    n = sum(len(s[1]) for s in systems)
    e = Engine(_params(case, systems[0][0]), case["precision"], max_particles=n,
               max_sims=len(systems))
    # the lists' best block size on this GPU; the defaults elsewhere
    e.set_tuning(pair_scheme=case["scheme"], block_size=256 if case["scheme"] == 2 else 128,
                 steps_per_graph=case["steps"])
    dim, dev = case["dim"], _device()

    def new(*shape):
        return torch.empty(shape, dtype=torch.float64, device=dev)

    out = {"r": new(n, dim), "v": new(n, dim), "u": new(n)}
    props = {k: new(n) for k in ("rho", "rho_lr", "t", "p", "pco", "udot")}
    props["vdot"] = new(n, dim)
    if case["heat"]:
        props["jq"] = new(n, dim)
    sims, at = [], 0
    for box, r, v, m, u in systems:
        sid = e.add(_params(case, box), r, v, m, u)
        sims.append((sid, (r, v, m, u), {k: x[at:at + len(r)] for k, x in out.items()}))
        at += len(r)
    return {"case": case, "engine": e, "sims": sims, "out": out, "props": props}


# ---- one pass --------------------------------------------------------------

def _as_computed(case, out):
    if case["precision"] == "fp64":
        return out
    cast = (lambda x: x.astype(np.float32)) if isinstance(out["vdot" if "vdot" in out else "v"],
                                                         np.ndarray) else torch.Tensor.float
    return {k: x if k == "r" else cast(x) for k, x in out.items()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "update":
        p = state["p"]
        p.r[:], p.v[:], p.m[:], p.u[:] = state["start"]
        p.run(DT, case["steps"])
        keys = ["r", "v", "u", "rho", "rho_lr", "t", "p", "pco", "vdot", "udot"]
        return _as_computed(case, {k: getattr(p, k) for k in keys + ["jq"] * case["heat"]})
    if kind == "pairs":
        nl = state["nl"]
        nl.build()
        return {"iap": nl.iap, "drij": nl.drij, "rsq": nl.rsq, "dv": nl.dv}
    if kind == "splat":
        s = state
        if case["dim"] == 2:
            return interpolate.splash_map_2d(s["x"], s["y"], s["r"], s["m"], s["rho"], s["a"],
                                             s["h"], s["bounds"], s["cutoff"])
        return interpolate.splash_map_3d(s["x"], s["y"], s["z"], s["r"], s["m"], s["rho"],
                                         s["a"], s["h"], s["bounds"], s["cutoff"])
    e = state["engine"]
    for sid, start, _ in state["sims"]:
        e.set_state(sid, *start)
    if kind == "eval":
        e.derivatives(state["sims"][0][0], out=state["props"])
        e.sync()
        return _as_computed(case, state["props"])
    e.advance(case["steps"])
    for sid, _, o in state["sims"]:
        e.get_state(sid, o["r"], o["v"], o["u"])
    out = dict(state["out"])
    if kind == "steps":
        e.properties(state["sims"][0][0], out=state["props"])
        out.update(state["props"])
    e.sync()
    return _as_computed(case, out)


# ---- the work of a pass ----------------------------------------------------

def work(case):
    dim = case["dim"]
    n = sum(math.prod(s) for s in _sim_sides(case))
    cut = _lengths(case)[2]
    ball = math.pi * cut ** 2 if dim == 2 else 4.0 / 3.0 * math.pi * cut ** 3
    pairs = 0.5 * n * case["density"] * ball
    state = 8.0 * (2 * dim + 2) * n
    if case["kind"] == "pairs":
        # in: r, v; out: two 8-byte indices, drij, rsq, dv of each pair
        ball = math.pi * (cut ** 2 + SKIN ** 2) if dim == 2 else \
            4.0 / 3.0 * math.pi * (cut ** 2 + SKIN ** 2) ** 1.5
        pairs = 0.5 * n * case["density"] * ball
        return {"bytes": 16.0 * dim * n + pairs * (16 + 8 * (2 * dim + 1)),
                "flops": pairs * (3 * dim - 1)}
    if case["kind"] == "splat":
        box = [k * case["density"] ** (-1.0 / dim) for k in (case["nx"], case["ny"])]
        k = [min(768, 2 * s + 1) for s in (case["nx"], case["ny"])]
        hs = _lengths({**case, "kernel": "lucy"})[0]
        # the particles of a 3D map that reach the plane
        reach = 1.0 if dim == 2 else min(
            1.0, 4.0 / 3.0 * hs / (case["nz"] * case["density"] ** (-1.0 / 3.0)))
        hits = n * reach * math.pi * hs ** 2 * k[0] * k[1] / (box[0] * box[1])
        return {"bytes": 8.0 * (n * (dim + 4) + k[0] * k[1] + k[0] + k[1]), "flops": 17.0 * hits}
    # flops of one unordered pair in one evaluation: density, force (14 of its
    # flops the viscosity's) and heat flux
    f = 3 * dim + 24 + 10 * dim + 42 - (0 if case["viscosity"] else 14)
    f += 10 * dim + 16 if case["heat"] else 0
    evals = 1 if case["kind"] == "eval" else case["steps"] * STAGES[case["integrator"]]
    size = 8 if case["precision"] == "fp64" else 4
    props = n * size * (6 + dim + (dim if case["heat"] else 0))
    if case["kind"] == "eval":
        byte = state + props
    elif case["kind"] == "batch":
        byte = state + 8.0 * (2 * dim + 1) * n
    else:
        byte = state + 8.0 * (2 * dim + 1) * n + props
    return {"bytes": byte, "flops": evals * pairs * f}


# ---- the same in plain 64-bit arithmetic -----------------------------------

def _kernel(case, h):
    """W(0) and the function r -> W, (dW/dr)/r."""
    dim, name, pi = case["dim"], case["kernel"], math.pi
    if name == "lucy":
        sig = 5 / (pi * h ** 2) if dim == 2 else 105 / (16 * pi * h ** 3)

        def fn(r):
            s = (1 - r / h).clamp_min(0.0)
            return sig * (1 + 3 * r / h) * s ** 3, -12 * sig / h ** 2 * s ** 2
        return sig, fn
    if name == "gaussian":
        sig = 1 / (h ** dim * pi ** (dim / 2))

        def fn(r):
            w = sig * torch.exp(-(r / h) ** 2)
            return w, -2 / h ** 2 * w
        return sig, fn
    if name == "debrun":
        sig = 10 / (pi * h ** 6) if dim == 2 else 15 / (pi * h ** 6)

        def fn(r):
            s = (h - r).clamp_min(0.0)
            return sig * s ** 3, -3 * sig * s ** 2 / r.clamp_min(1e-300)
        return sig * h ** 3, fn
    sig = 10 / (7 * pi * h ** 2) if dim == 2 else 1 / (pi * h ** 3)

    def fn(r):
        q = r / h
        s = (2 - q).clamp_min(0.0)
        inner = q < 1
        w = torch.where(inner, 1 - 1.5 * q ** 2 + 0.75 * q ** 3, 0.25 * s ** 3)
        g = torch.where(inner, -3 + 2.25 * q, -0.75 * s ** 2 / q.clamp_min(1e-300))
        return sig * w, sig / h ** 2 * g
    return sig, fn


def _image(d, box):
    L = torch.tensor(box, dtype=torch.float64, device=d.device)
    return torch.where(d > L / 2, d - L, torch.where(d < -L / 2, d + L, d))


def _neighbours(r, box, thr):
    """[n, k] neighbour indices (rsq < thr), -1 where a particle has fewer."""
    n, dim = r.shape
    dev = r.device
    rc = math.sqrt(thr) * (1 + 1e-9)
    nc = [int(L // rc) for L in box]
    rows, cols = [], []
    if min(nc) < 3:      # a small box: every pair
        per = max(1, int(4e7 // n))
        for b in range(0, n, per):
            d = _image(r[None, :, :] - r[b:b + per, None, :], box)
            hit = (d * d).sum(-1) < thr
            hit[torch.arange(hit.shape[0], device=dev), torch.arange(b, b + hit.shape[0],
                                                                     device=dev)] = False
            i, j = hit.nonzero(as_tuple=True)
            rows.append(i + b)
            cols.append(j)
    else:
        L = torch.tensor(box, dtype=torch.float64, device=dev)
        k = torch.tensor(nc, device=dev)
        cell = torch.minimum((torch.remainder(r, L) / (L / k)).long(), k - 1)
        lin = torch.zeros(n, dtype=torch.long, device=dev)
        for a in range(dim):
            lin = lin * nc[a] + cell[:, a]
        ncell = math.prod(nc)
        order = torch.argsort(lin)
        count = torch.bincount(lin, minlength=ncell)
        start = torch.cumsum(count, 0) - count
        pad = int(count.max())
        table = torch.full((ncell, pad), n, dtype=torch.long, device=dev)
        table[lin[order], torch.arange(n, device=dev) - start[lin[order]]] = order
        off = torch.stack(torch.meshgrid(*[torch.arange(-1, 2, device=dev)] * dim,
                                         indexing="ij"), -1).reshape(-1, dim)
        rx = torch.cat([r, torch.full((1, dim), 1e30, device=dev, dtype=torch.float64)])
        per = max(1, int(6e7 // (pad * pad * len(off))))
        for b in range(0, ncell, per):
            c = torch.arange(b, min(ncell, b + per), device=dev)
            xyz, rest = [], c
            for a in reversed(range(dim)):
                xyz.insert(0, rest % nc[a])
                rest = rest // nc[a]
            near = torch.zeros(len(c), len(off), dtype=torch.long, device=dev)
            for a in range(dim):
                near = near * nc[a] + (xyz[a][:, None] + off[None, :, a]) % nc[a]
            cand = table[near].reshape(len(c), -1)
            own = table[c]
            rsq = 0.0
            for a in range(dim):
                d = rx[cand, a][:, None, :] - rx[own, a][:, :, None]
                d = torch.where(d > box[a] / 2, d - box[a],
                                torch.where(d < -box[a] / 2, d + box[a], d))
                rsq = rsq + d * d
            hit = (rsq < thr) & (cand[:, None, :] != own[:, :, None]) & (own[:, :, None] < n) & (
                cand[:, None, :] < n)
            q, i, j = hit.nonzero(as_tuple=True)
            rows.append(own[q, i])
            cols.append(cand[q, j])
            del rsq, hit, d
    i, j = torch.cat(rows), torch.cat(cols)
    del rows, cols
    count = torch.bincount(i, minlength=n)
    # rows come in runs of one particle; its first entry is where its run starts
    first = torch.zeros(n, dtype=torch.long, device=dev)
    new = torch.ones(len(i), dtype=torch.bool, device=dev)
    new[1:] = i[1:] != i[:-1]
    first[i[new]] = new.nonzero(as_tuple=True)[0]
    out = torch.full((n, max(1, int(count.max()))), -1, dtype=torch.int32, device=dev)
    out[i, torch.arange(len(i), device=dev) - first[i]] = j.int()
    return out


def _rates(case, box, r, v, m, u):
    """One evaluation: rho, rho_lr, t, p, pco, vdot, udot, jq."""
    n, dim = r.shape
    hs, hl, cut = _lengths(case)
    w0s, ks = _kernel(case, hs)
    w0l, kl = _kernel(case, hl)
    nb = _neighbours(r, box, cut * cut)
    per = max(1, int(3e7 // nb.shape[1]))

    def chunks():
        for b in range(0, n, per):
            j = nb[b:b + per].long()
            live = j >= 0
            j = j.clamp_min(0)
            d = _image(r[j] - r[b:b + per, None, :], box)
            rsq = (d * d).sum(-1)
            yield slice(b, b + per), j, live.to(torch.float64), d, rsq, rsq.sqrt()

    rho, rhol = torch.full_like(u, w0s), torch.full_like(u, w0l)
    for s, j, live, d, rsq, dist in chunks():
        rho[s] += (m[j] * live * ks(dist)[0]).sum(1)
        rhol[s] += (m[j] * live * kl(dist)[0]).sum(1)
    t = ((u + A * rho) / KB).clamp_min(0.0)
    p = rho * KB * t / (1 - B * rho)
    pco = -A * rhol ** 2
    jq = torch.zeros_like(r)
    if case["heat"]:
        for s, j, live, d, rsq, dist in chunks():
            f = live * m[j] / rho[j] * (t[j] - t[s, None]) * ks(dist)[1]
            jq[s] = (f[..., None] * d).sum(1)
    vdot, udot = torch.zeros_like(r), torch.zeros_like(u)
    for s, j, live, d, rsq, dist in chunks():
        gs, gl = ks(dist)[1] * live, kl(dist)[1] * live
        dv = ((v[j] - v[s, None, :]) * d).sum(-1)
        f = p[s, None] / rho[s, None] ** 2 + p[j] / rho[j] ** 2
        if case["viscosity"]:
            mu = hs * dv / (rsq + EPS * hs * hs)
            pi = (-ALPHA * mu + BETA * mu * mu) / (0.5 * (rho[s, None] + rho[j]))
            f = f + torch.where(dv < 0, pi, torch.zeros_like(pi))
        a = f * gs + (pco[s, None] / rhol[s, None] ** 2 + pco[j] / rhol[j] ** 2) * gl
        vdot[s] = (a[..., None] * d).sum(1)
        du = 0.5 * a * dv * m[j]
        if case["heat"]:
            q = jq[s, None, :] / rho[s, None, None] ** 2 + jq[j] / rho[j][..., None] ** 2
            du = du - m[j] * (q * d).sum(-1) * gs
        udot[s] = du.sum(1)
    return {"rho": rho, "rho_lr": rhol, "t": t, "p": p, "pco": pco, "vdot": vdot, "udot": udot,
            "jq": jq}


def _steps(case, box, r, v, m, u):
    first = last = None
    for _ in range(case["steps"]):
        def f(rr, vv, uu):
            nonlocal first, last
            last = _rates(case, box, rr, vv, m, uu)
            first = first or last
            return vv, last["vdot"], last["udot"]
        first, x = None, (r, v, u)

        def add(x, k, c):
            return [a + c * b for a, b in zip(x, k)]
        k1 = f(*x)
        if case["integrator"] == "euler":
            x = add(x, k1, DT)
        elif case["integrator"] == "ieuler":
            k2 = f(*add(x, k1, DT))
            x = add(add(x, k1, DT / 2), k2, DT / 2)
        else:
            k2 = f(*add(x, k1, DT / 2))
            k3 = f(*add(x, k2, DT / 2))
            k4 = f(*add(x, k3, DT))
            for k, c in ((k1, 1), (k2, 2), (k3, 2), (k4, 1)):
                x = add(x, k, c * DT / 6)
        r, v, u = x
        L = torch.tensor(box, dtype=torch.float64, device=r.device)
        r = torch.where(r > L, torch.zeros_like(r), torch.where(r < 0, L.expand_as(r), r))
        if case["thermostat"]:
            last = dict(last, t=last["t"] * (TEMP / last["t"].mean()))
            u = KB * last["t"] - A * first["rho"]
    out = {"r": r, "v": v, "u": u}
    # rho, p and pco are those of the step's first evaluation
    out.update(last, rho=first["rho"], p=first["p"], pco=first["pco"])
    return out


def exact(case, seed):
    kind, dim = case["kind"], case["dim"]
    if kind == "splat":
        return _exact_splat(case, seed)
    systems = _systems(case, seed)
    box, r, v, m, u = systems[0]
    if kind == "pairs":
        cut = _lengths(case)[2]
        r, v = _numbered(case, seed)
        nb = _neighbours(r, box, cut * cut + SKIN * SKIN).long()
        i = torch.arange(len(r), device=r.device)[:, None].expand_as(nb)
        i, j = i[nb > i], nb[nb > i]
        at = torch.argsort(i * len(r) + j)
        i, j = i[at], j[at]
        d = _image(r[j] - r[i], box)
        return {"iap": None, "drij": d, "rsq": (d * d).sum(-1), "dv": v[j] - v[i]}
    if kind == "eval":
        out = _rates(case, box, r, v, m, u)
    elif kind == "batch":
        got = [_steps(case, *s) for s in systems]
        out = {k: torch.cat([g[k] for g in got]) for k in ("r", "v", "u")}
    else:
        out = _steps(case, box, r, v, m, u)
    if not case["heat"]:
        out.pop("jq", None)
    return out


def _exact_splat(case, seed):
    s = prepare(case, seed)
    dim, dev = case["dim"], _device()
    r, m, rho, a, h, x, y = [torch.tensor(s[k], device=dev, dtype=torch.float64)
                             for k in ("r", "m", "rho", "a", "h", "x", "y")]
    cut, (x0, x1, y0, y1) = s["cutoff"], s["bounds"]
    dz = r[:, 2] - s["z"] if dim == 3 else torch.zeros_like(m)
    res = x[1] - x[0]
    xa, ya = (torch.floor((r[:, k] - cut - lo) / res).long() for k, lo in ((0, x0), (1, y0)))
    xb, yb = (torch.floor((r[:, k] + cut - lo) / res).long() for k, lo in ((0, x0), (1, y0)))
    Z = torch.zeros(len(x) * len(y), dtype=torch.float64, device=dev)
    for p in range(int((xb - xa).max())):
        for q in range(int((yb - ya).max())):
            xx, yy = xa + p, ya + q
            ok = (xx < xb) & (yy < yb) & (dz <= cut)
            xx = torch.where(xx >= len(x), xx - len(x), torch.where(xx < 0, xx + len(x), xx))
            yy = torch.where(yy >= len(y), yy - len(y), torch.where(yy < 0, yy + len(y), yy))
            ok &= (xx >= 0) & (xx < len(x)) & (yy >= 0) & (yy < len(y))
            xx, yy = xx.clamp(0, len(x) - 1), yy.clamp(0, len(y) - 1)
            d = torch.stack([r[:, 0] - x[xx], y[yy] - r[:, 1]], dim=1)
            d = _image(d, [x1, y1])
            rsq = (d * d).sum(1) + dz * dz
            sig = 105 / (16 * math.pi * h ** 3) if dim == 3 else 5 / (math.pi * h ** 2)
            t = (1 - rsq.sqrt() / h).clamp_min(0.0)
            w = a * m / rho * sig * (1 + 3 * rsq.sqrt() / h) * t ** 3
            ok &= rsq < cut * cut
            Z.index_add_(0, (xx * len(y) + yy)[ok], w[ok])
    return Z.reshape(len(x), len(y))
