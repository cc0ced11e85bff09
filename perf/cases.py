"""Performance cases of the mover + P2G framework, called as a user's program calls it.

A case names the call ("kind") and its sizes:

* ``mover``         GridContext.set_fields + mover: the plain push over one batch of particles
* ``deposit``       GridContext.p2g + apply_bc_ids per species: the plain moments
* ``mover_interp``  GridContext.set_fields + mover_interp + apply_bc_ids: push and deposit in one call
* ``sim``           Simulation.set_fields + cycle + moments: one cycle of the precision form
* ``hat``           hat_densities: the field solver's source terms from the moments
* ``driver``        the drop-in calls over the reference's structs, particles resident: mover_PC (and
                    particle_sort) per species, then the moment section in one call
* ``serve``         Server: a few independent jobs, from submission to their moments

The inputs are the repository's seeded GEM workloads. The electric field of the 0.15625 cells is the
GEM workload's noise, with the other sign in every second pass, as a solver hands over new fields
each cycle (one field kept for ever would pile the electrons up in its sinks). Particles pushed in
place come in several batches, the next one in each pass, so that a batch stays near the order it
was made in however many passes are timed.
"""
from __future__ import annotations

import math
import weakref

import numpy as np
import torch

from sputnipic_b200 import device, dropin, hat
from sputnipic_b200 import workload as W
from sputnipic_b200.serve import Job, Server
from sputnipic_b200.sim import Simulation

PERIODIC = {"gem": (True, False, True), "periodic": (True, True, True),
            "walls": (False, False, False)}
KEYS = "xyzuvw"


def listed():
    return [
        # the GEM benchmark's electrons, 65.5M in cell order: the largest push
        _case("mover_gem", "mover", 128, 64, 64, 125, species=0),
        # an odd grid between walls, electrons that have left the cells they were last sorted by
        _case("mover_drifted", "mover", 61, 45, 33, 27, species=0, bc="walls", order="drifted"),
        # the small GEM cycle's moments, four species: launches and latency
        _case("deposit_small", "deposit", 32, 16, 16, 27, ns=4, cell=0.625),
        # one GEM species' moments, 65.5M particles in cell order
        _case("deposit_gem", "deposit", 128, 64, 64, 125, ns=1),
        # an odd periodic grid, particles some cycles after the last sort
        _case("deposit_drifted", "deposit", 61, 45, 33, 27, ns=2, bc="periodic", order="drifted"),
        # mover_interp of ions on an odd grid
        _case("mover_interp_ragged", "mover_interp", 101, 47, 53, 27, species=1),
        # the small GEM cycle in the precision form: launches and latency
        _case("sim_small", "sim", 32, 16, 16, 27, ns=4, cell=0.625),
        # the headline workload: 4 x 65.5M particles
        _case("sim_gem", "sim", 128, 64, 64, 125, ns=4),
        # the same grid at 8 particles per cell, where the grid's share is large
        _case("sim_sparse", "sim", 128, 64, 64, 8, ns=4),
        # the solver's source terms on the GEM grid in double precision
        _case("hat_gem", "hat", 128, 64, 64, 1, ns=4, fp=64),
        # a cycle of the reference's driver in which it sorts, on an odd grid
        _case("driver_sort", "driver", 61, 45, 33, 27, ns=4, sort=True),
        # four test-particle jobs of different grids at once
        _case("serve_mix", "serve", 64, 32, 32, 16, ns=2, jobs=4, cycles=8),
    ]


def _case(name, kind, nx, ny, nz, ppc, **kw):
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "ppc": ppc, "bc": "gem", "cell": 0.15625}
    c.update(kw)
    if name:
        c["name"] = name
    if kind in ("mover", "deposit", "mover_interp"):
        c.setdefault("order", "cells")
    if kind == "sim":
        c.setdefault("deterministic", False)
    return c


def draw(rng):
    kind = rng.choice(("mover", "deposit", "mover_interp", "sim", "hat", "driver", "serve"))
    bc = rng.choice(sorted(PERIODIC))
    order = rng.choice(("cells", "drifted"))

    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    def sizes(cells, unit):
        """Three extents near the cube root of `cells`, multiples of `unit`."""
        side = cells ** (1 / 3)
        return [max(2, round(side * rng.uniform(0.6, 1.6) / u)) * u for u in unit]

    if kind == "hat":
        return _case(None, kind, *sizes(log(4e3, 5e5), (1, 1, 1)), 1, bc=bc, ns=rng.randint(1, 6),
                     fp=rng.choice((32, 64)))
    if kind == "serve":
        ppc = round(log(4, 20), 1)
        return _case(None, kind, *sizes(log(2e3, 4e4), (4, 4, 4)), ppc, bc=bc,
                     ns=rng.choice((2, 4)), jobs=rng.randint(2, 4), cycles=rng.randint(2, 8))
    ppc = round(log(4, 125), 1)
    n = log(2e4, 5e6 if kind == "driver" else 2.5e7)   # particles of a species
    unit = (8, 4, 4) if kind == "sim" else (1, 1, 1)
    nx, ny, nz = sizes(min(max(n / ppc, 1e3), 6e5), unit)
    if kind in ("mover", "mover_interp"):
        return _case(None, kind, nx, ny, nz, ppc, species=rng.randint(0, 3), bc=bc, order=order)
    if kind == "deposit":
        return _case(None, kind, nx, ny, nz, ppc, ns=rng.randint(1, 4), bc=bc, order=order)
    if kind == "sim":
        return _case(None, kind, nx, ny, nz, ppc, ns=rng.randint(1, 4), bc=bc,
                     deterministic=rng.random() < 0.25)
    return _case(None, kind, nx, ny, nz, ppc, ns=rng.choice((2, 4)), bc=bc,
                 sort=rng.random() < 0.5)


# --- inputs --------------------------------------------------------------------------------------
def _workload(c, seed, n=None):
    nx, ny, nz = n or (c["nx"], c["ny"], c["nz"])
    d = c["cell"]
    return W.GemWorkload(name="case", nxc=nx, nyc=ny, nzc=nz, Lx=nx * d, Ly=ny * d, Lz=nz * d,
                         periodic=PERIODIC[c["bc"]], E_amp=1e-3 if d < 0.5 else 0.0,
                         lattice=5 if c["ppc"] == 125 else 0, seed=seed % (1 << 31),
                         species=W.gem_species((c["ppc"],) * 4))


def _fields(wl):
    """The fields of even and of odd passes."""
    F = device.gen_fields(wl)
    return F, [-f for f in F[:3]] + F[3:]


def _particles(c, wl, s):
    p = device.gen_particles(wl, s)
    if c.get("order") == "drifted":
        # the order of the cells that the particles were in when the arrays were last sorted
        g = torch.Generator(device="cuda").manual_seed(wl.seed * 8 + s)
        key = torch.zeros(p["x"].numel(), dtype=torch.int64, device="cuda")
        for k, n, far in zip("xyz", (wl.nxc, wl.nyc, wl.nzc), (1.5, 0.25, 1.5)):
            was = p[k] / c["cell"] + far * torch.randn(p[k].numel(), generator=g, device="cuda")
            key = key * n + was.floor().long().clamp(0, n - 1)
        order = torch.argsort(key, stable=True)
        p = {k: p[k][order] for k in "xyzuvwq"}
    return p


def _batches(c, seed):
    """How many batches a program that pushes them in turn holds."""
    n = c["nx"] * c["ny"] * c["nz"] * c["ppc"]
    return [seed + 7919 * k for k in range(max(2, min(48, int(24e9 / (28 * n)))))]


def _job_cases(c, seed):
    """A serving batch: jobs of the case's grid, of half and of twice its x extent."""
    out = []
    for k in range(c["jobs"]):
        f = (1.0, 0.5, 2.0)[k % 3]
        nx = max(4, int(c["nx"] * f) // 4 * 4)
        out.append((_workload(c, seed + 31 * k, (nx, c["ny"], c["nz"])), c["cycles"] + k % 4))
    return out


_live = weakref.WeakSet()   # states that hold drop-in mirrors


class _State(dict):
    __hash__ = object.__hash__


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def prepare(case, seed):
    c, st = case, _State(case=case, k=0)
    kind = c["kind"]
    if kind == "hat":
        wl = _workload(c, seed)
        g = torch.Generator(device="cuda").manual_seed(wl.seed)
        dt = torch.float64 if c["fp"] == 64 else torch.float32
        cells = (wl.nxc + 2) * (wl.nyc + 2) * (wl.nzc + 2)

        def normal(n, sc):
            return torch.randn(n, generator=g, device="cuda", dtype=dt) * sc
        st["mom"] = [[normal(wl.nodes, sc) for sc in (1.0,) + (1e-2,) * 3 + (1e-3,) * 6]
                     for _ in range(c["ns"])]
        st["B"] = [normal(wl.nodes, 0.03) for _ in range(3)]
        st["rhoc"] = normal(cells, 1.0)
        st["desc"] = hat.hat_desc(wl, qom=_hat_qom(c["ns"]), fp=c["fp"])
        return st
    if kind == "serve":
        st["jobs"] = [Job(wl, device.gen_fields(wl), [_particles(c, wl, s) for s in range(c["ns"])],
                          n) for wl, n in _job_cases(c, seed)]
        st["server"] = Server(hbm_budget=16 << 30, reserve_bytes=4 << 30)
        torch.cuda.synchronize()   # the engine reads the inputs on streams of its own
        return st
    wl = st["wl"] = _workload(c, seed)
    st["F"] = _fields(wl)
    if kind == "driver":
        if not _live:
            dropin.release_all()
            dropin.set_residency(True)
        _live.add(st)
        st["param"] = dropin.make_parameters(wl, ns=c["ns"])
        st["param"].sort_cps = 2
        st["grd"] = dropin.setGrid(st["param"])
        st["F"] = [dropin.field_allocate(st["grd"], [_pinned(f) for f in F]) for F in st["F"]]
        st["parts"] = []
        for s in range(c["ns"]):
            a = {k: _pinned(v) for k, v in _particles(c, wl, s).items()}
            st["parts"].append(dropin.particle_allocate(st["param"], s, arrays=a))
            dropin.invalidate_particles(st["parts"][-1])
        st["ids"] = [dropin.interp_dens_species_allocate(st["grd"], s) for s in range(c["ns"])]
        st["idn"] = dropin.interp_dens_net_allocate(st["grd"])
        return st
    if kind == "sim":
        st["sim"] = sim = Simulation(wl, species=range(c["ns"]), graph=True,
                                     deterministic=c["deterministic"])
        sim.set_fields(st["F"][0])
        for s in range(c["ns"]):
            sim.load_species(s, _particles(c, wl, s))
        torch.cuda.synchronize()
        return st
    st["ctx"] = device.GridContext(wl)
    if kind == "deposit":
        st["parts"] = [_particles(c, wl, s) for s in range(c["ns"])]
        st["mom"] = [torch.zeros(10, wl.nodes, device="cuda") for _ in range(c["ns"])]
        return st
    st["push"] = device.push_params(wl, c["species"])
    st["parts"] = [_particles(c, wl.with_(seed=b % (1 << 31)), c["species"])
                   for b in _batches(c, seed)]
    if kind == "mover_interp":
        st["mom"] = [torch.zeros(10, wl.nodes, device="cuda")]
    return st


def _hat_qom(ns):
    return [(-64.0, 1.0)[s % 2] for s in range(ns)]


# --- one pass --------------------------------------------------------------------------------------
def _groups(mom):
    """rhon, J and the pressures apart: their magnitudes differ."""
    return [mom[0], mom[1:4], mom[4:10]]


def _fold(wl, mom):
    """applyBCids on raw moments: periodic planes folded, the others doubled."""
    m = mom.view(10, wl.nxn, wl.nyn, wl.nzn)
    inner = m[:, 1:-1, 1:-1, 1:-1]
    for fold in (True, False):
        for a in range(3):
            if wl.periodic[a] != fold:
                continue
            lo, hi = inner.select(a + 1, 0), inner.select(a + 1, -1)
            if fold:
                both = lo + hi
                lo.copy_(both)
                hi.copy_(both)
            else:
                lo.mul_(2)
                hi.mul_(2)
    return mom


def run(st):
    c, k = st["case"], st["k"]
    st["k"] = k + 1
    kind = c["kind"]
    if kind == "hat":
        return hat.hat_densities(st["desc"], st["mom"], st["B"], st["rhoc"])
    if kind == "serve":
        srv, out = st["server"], {}
        ids = {srv.submit(j): i for i, j in enumerate(st["jobs"])}
        while ids:
            srv.step()
            for jid in srv.finished():
                i = ids.pop(jid)
                j = st["jobs"][i]
                for s in range(c["ns"]):
                    r = srv.result(jid, s, j.parts[s]["x"].numel(), j.wl.nodes, particles=False)
                    out[i, s] = _fold(j.wl, r["moments"])
                srv.release(jid)
        # the moments of the jobs side by side, species by species
        return [[torch.cat([g.reshape(-1) for g in gs]) for gs in
                 zip(*(_groups(out[i, s]) for i in range(len(st["jobs"]))))]
                for s in range(c["ns"])]
    wl, F = st["wl"], st["F"][k % 2]
    if kind == "driver":
        for p in st["parts"]:
            dropin.mover_PC(p, F, st["grd"], st["param"], raise_on_error=True)
            if c["sort"]:
                dropin.particle_sort(st["param"], p, st["grd"], raise_on_error=True)
        dropin.interp_all_species(st["parts"], st["ids"], st["idn"], st["grd"], st["param"],
                                  raise_on_error=True)
        return [dropin.moments(i) for i in st["ids"]] + [
            [st["idn"]._arrays[m] for m in dropin.MOMENT_NAMES]]
    if kind == "sim":
        sim = st["sim"]
        sim.set_fields(F)
        sim.cycle(1)
        return [_groups(sim.moments(s, bc=True)) for s in range(c["ns"])]
    ctx = st["ctx"]
    if kind == "deposit":
        for p, m in zip(st["parts"], st["mom"]):
            m.zero_()
            ctx.p2g(p, m)
            ctx.apply_bc_ids(m, wl.periodic)
        return [_groups(m) for m in st["mom"]]
    p = st["parts"][k % len(st["parts"])]
    ctx.set_fields(F)
    if kind == "mover":
        ctx.mover(p, st["push"])
        return [p[a] for a in KEYS]
    m = st["mom"][0]
    m.zero_()
    ctx.mover_interp(p, st["push"], m)
    ctx.apply_bc_ids(m, wl.periodic)
    return [p[a] for a in KEYS], _groups(m)


# --- what a pass cannot do without --------------------------------------------------------------------
def work(case):
    c = case
    nodes = (c["nx"] + 3) * (c["ny"] + 3) * (c["nz"] + 3)
    n = c["nx"] * c["ny"] * c["nz"] * c["ppc"]
    ns = c.get("ns", 1)
    push, dep = 520, 190   # operations per particle: three gathers and solves; 80 terms
    kind = c["kind"]
    if kind == "mover":
        return {"bytes": 48 * n + 24 * nodes, "flops": push * n}
    if kind == "deposit":
        return {"bytes": ns * (28 * n + 40 * nodes), "flops": ns * dep * n}
    if kind == "mover_interp":
        return {"bytes": 52 * n + 64 * nodes, "flops": (push + dep) * n}
    if kind == "sim":
        return {"bytes": ns * (52 * n + 80 * nodes) + 24 * nodes, "flops": ns * (push + dep) * n}
    if kind == "driver":   # x..q read, x..w written; a sorting cycle writes q too
        return {"bytes": ns * ((56 if c["sort"] else 52) * n + 40 * nodes) + 64 * nodes,
                "flops": ns * (push + dep) * n}
    if kind == "hat":
        b = c["fp"] // 8
        cells = (c["nx"] + 2) * (c["ny"] + 2) * (c["nz"] + 2)
        return {"bytes": b * ((9 * ns + 6) * nodes + 2 * cells), "flops": (ns * 200 + 80) * nodes}
    total = {"bytes": 0.0, "flops": 0.0}
    for wl, cycles in _job_cases(c, 0):
        m = wl.cells * c["ppc"] * ns
        total["bytes"] += (28 + 52 * cycles) * m + (24 + 80 * ns) * wl.nodes
        total["flops"] += cycles * (push + dep) * m
    return total


def tolerance(case):
    kind = case["kind"]
    if kind in ("mover", "hat"):
        return "exact"   # the reference's operations, one by one
    # sums of FP32 terms in any order; measured over runs of the same inputs (rel, max): sim 2.3e-7,
    # 2.2e-6; deposits 1.3e-7, 2.2e-6; driver 1.9e-6, 1.8e-5 (each moment on its own, and the
    # off-diagonal pressures cancel); serve as sim, over several cycles
    if kind == "driver":
        return {"rel": 1e-5, "max": 1e-4}
    if kind == "serve":
        return {"rel": 2e-6, "max": 2e-5}
    return {"rel": 1e-6, "max": 1e-5}


# --- the same in 64 bits ---------------------------------------------------------------------------
def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "hat":
        return _hat64(c, prepare(case, seed))
    if kind == "serve":
        per = [[] for _ in range(c["ns"])]
        for wl, cycles in _job_cases(c, seed):
            F = _stack64(device.gen_fields(wl))
            for s in range(c["ns"]):
                p = _particles(c, wl, s)
                for _ in range(cycles):
                    p = dict(zip(KEYS, _push64(wl, F, p, wl.species[s].qom)), q=p["q"])
                per[s].append(_groups(_fold(wl, _deposit64(wl, p))))
        return [[torch.cat([g.reshape(-1) for g in gs]) for gs in zip(*js)] for js in per]
    wl = _workload(c, seed)
    F = _stack64(_fields(wl)[0])
    if kind == "mover":
        return _push64(wl, F, _particles(c, wl, c["species"]), wl.species[c["species"]].qom)
    if kind == "mover_interp":
        p = _particles(c, wl, c["species"])
        p.update(zip(KEYS, _push64(wl, F, p, wl.species[c["species"]].qom)))
        return [p[a] for a in KEYS], _groups(_fold(wl, _deposit64(wl, p)))
    moms = []
    for s in range(c["ns"]):
        p = _particles(c, wl, s)
        if kind != "deposit":
            p.update(zip(KEYS, _push64(wl, F, p, wl.species[s].qom)))
        moms.append(_fold(wl, _deposit64(wl, p)))
    if kind == "driver":
        return [list(m.cpu()) for m in moms + [sum(moms)]]
    return [_groups(m) for m in moms]


CHUNK = 1 << 22


def _stack64(F):
    return torch.stack([f.double() for f in F], 1)


def _push64(wl, F, p, qom):
    """mover_PC in double precision: three predictor-corrector steps, the particle boundaries."""
    n = p["x"].numel()
    out = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(6)]
    for a in range(0, n, CHUNK):
        got = _push64_some(wl, F, [p[k][a:a + CHUNK].double() for k in KEYS], qom)
        for o, v in zip(out, got):
            o[a:a + CHUNK] = v
    return out


def _push64_some(wl, F, p, qom):
    d = (wl.dx, wl.dy, wl.dz)
    x0, v0 = torch.stack(p[:3], 1), torch.stack(p[3:], 1)
    dt, h = wl.dt, qom * 0.5 * wl.dt / wl.c
    D = torch.tensor(d, dtype=torch.float64, device="cuda")
    x = x0
    for _ in range(wl.niter):
        i = 2 + (x / D).trunc()
        f = x / D - (i - 2)
        i = i.long()
        base = (i[:, 0] * wl.nyn + i[:, 1]) * wl.nzn + i[:, 2]
        EB = torch.zeros(x.shape[0], 6, dtype=torch.float64, device="cuda")
        for a in (0, 1):
            for b in (0, 1):
                for e in (0, 1):   # a, b, e = 1: the lower node of the axis
                    w = ((1 - f[:, 0] if a else f[:, 0]) * (1 - f[:, 1] if b else f[:, 1])
                         * (1 - f[:, 2] if e else f[:, 2]))
                    EB += w[:, None] * F[base - (a * wl.nyn + b) * wl.nzn - e]
        E, B = EB[:, :3], EB[:, 3:]
        t = v0 + h * E
        v = (t + h * (torch.linalg.cross(t, B) + h * (t * B).sum(1, keepdim=True) * B)) / (
            1 + h * h * (B * B).sum(1, keepdim=True))
        x = x0 + v * (0.5 * dt)
    x, v = x0 + v * dt, 2 * v - v0
    for a, L in enumerate((wl.Lx, wl.Ly, wl.Lz)):
        X, V = x[:, a], v[:, a]
        for out, back in ((X > L, lambda q: q - L if wl.periodic[a] else 2 * L - q),
                          (None, lambda q: q + L if wl.periodic[a] else -q)):
            out = X < 0 if out is None else out
            X = torch.where(out, back(X), X)
            if not wl.periodic[a]:
                V = torch.where(out, -V, V)
        x[:, a], v[:, a] = X, V
    return [x[:, a] for a in range(3)] + [v[:, a] for a in range(3)]


def _deposit64(wl, p):
    """interpP2G in double precision: ten moments on the nodes."""
    mom = torch.zeros(wl.nodes, 10, dtype=torch.float64, device="cuda")
    vol = wl.dx * wl.dy * wl.dz
    for s in range(0, p["x"].numel(), CHUNK):
        x, y, z, u, v, w, q = (p[k][s:s + CHUNK].double() for k in "xyzuvwq")
        r = [x / wl.dx, y / wl.dy, z / wl.dz]
        i = [t.floor() for t in r]
        f = [t - k for t, k in zip(r, i)]
        base = ((i[0].long() + 2) * wl.nyn + i[1].long() + 2) * wl.nzn + i[2].long() + 2
        terms = torch.stack([torch.ones_like(u), u, v, w, u * u, u * v, u * w, v * v, v * w, w * w],
                            1) * (q / vol)[:, None]
        for a in (0, 1):
            for b in (0, 1):
                for e in (0, 1):
                    wgt = ((1 - f[0] if a else f[0]) * (1 - f[1] if b else f[1])
                           * (1 - f[2] if e else f[2]))
                    mom.index_add_(0, base - (a * wl.nyn + b) * wl.nzn - e, wgt[:, None] * terms)
    return mom.T.contiguous()


def _fill64(a, s, per, yhi):
    """Guard cells of a scalar array: periodic faces, edges and corners, then the other faces."""
    e = [n - 1 for n in a.shape]

    def src(x, ax):
        return s if x == e[ax] else e[ax] - s

    inner = [slice(1, n) for n in e]
    for ax in range(3):
        if per[ax]:
            for g in (0, e[ax]):
                at, fr = list(inner), list(inner)
                at[ax], fr[ax] = g, src(g, ax)
                a[tuple(at)] = a[tuple(fr)].clone()
    for ax in range(3):
        o = [k for k in range(3) if k != ax]
        if per[o[0]] or per[o[1]]:
            along = slice(1, yhi) if ax == 1 else inner[ax]
            for g in (0, e[o[0]]):
                for h in (0, e[o[1]]):
                    at, fr = [along] * 3, [along] * 3
                    at[o[0]], at[o[1]] = g, h
                    fr[o[0]], fr[o[1]] = src(g, o[0]), src(h, o[1])
                    a[tuple(at)] = a[tuple(fr)].clone()
    if any(per):
        for g in (0, e[0]):
            for h in (0, e[1]):
                for k in (0, e[2]):
                    a[g, h, k] = a[src(g, 0), src(h, 1), src(k, 2)].clone()
    for ax in range(3):
        if not per[ax]:
            a.select(ax, 0).copy_(a.select(ax, 1).clone())
            a.select(ax, e[ax]).copy_(a.select(ax, e[ax] - 1).clone())
    return a


def _diff64(a, ax, inv):
    """Derivative of a node array along `ax` on the inner cells."""
    d = a.narrow(ax, 1, a.shape[ax] - 1) - a.narrow(ax, 0, a.shape[ax] - 1)
    for o in range(3):
        if o != ax:
            d = d.narrow(o, 1, d.shape[o] - 1) + d.narrow(o, 0, d.shape[o] - 1)
    return (0.25 * inv) * d[1:-1, 1:-1, 1:-1]


def _hat64(c, st):
    wl, d = _workload(c, 0), st["desc"]
    node, cell = (wl.nxn, wl.nyn, wl.nzn), (wl.nxc + 2, wl.nyc + 2, wl.nzc + 2)
    inv, per = (d.invdx, d.invdy, d.invdz), wl.periodic
    B = torch.stack([b.double().view(node) for b in st["B"]])
    J = torch.zeros((3,) + node, dtype=torch.float64, device="cuda")
    for s in range(c["ns"]):
        m = [t.double().view(node) for t in st["mom"][s]]
        rows = ((4, 5, 6), (5, 7, 8), (6, 8, 9))
        T = torch.stack(m[1:4])
        for r in range(3):
            t = torch.zeros(cell, dtype=torch.float64, device="cuda")
            t[1:-1, 1:-1, 1:-1] = (-0.5 * d.dt) * sum(
                _diff64(m[rows[r][ax]], ax, inv[ax]) for ax in range(3))
            _fill64(t, 1, per, wl.nyn - 1)
            for ax in range(3):
                t = t.narrow(ax, 1, t.shape[ax] - 1) + t.narrow(ax, 0, t.shape[ax] - 1)
            T[r, 1:-1, 1:-1, 1:-1] += 0.125 * t
        o = (0.5 * _hat_qom(c["ns"])[s] * d.dt / d.c) * B
        J += (T + torch.linalg.cross(T, o, dim=0) + (T * o).sum(0) * o) / (1 + (o * o).sum(0))
    for r in range(3):
        _fill64(J[r], 2, per, wl.nyn - 1)
    rho = st["rhoc"].double().view(cell).clone()
    rho[1:-1, 1:-1, 1:-1] -= d.dt * d.th * sum(_diff64(J[ax], ax, inv[ax]) for ax in range(3))
    _fill64(rho, 1, per, wl.nyn - 1)
    return tuple(J[r].reshape(-1) for r in range(3)) + (rho.reshape(-1),)
