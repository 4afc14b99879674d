"""The work a user has this framework do, as timed cases.

A pass is one output interval of a program: it steps the runs it keeps and reads what
it plots or writes at the end of the interval (the fields of the mesh, for discharges
the collision and wall counts too), or runs swarm requests and reads their results.
Sizes are those of the benchmark's decks and of the tests, and the ranges between them.

  sim1d   1D discharges and instabilities (Simulation1D): the two-stream and Landau
          decks (periodic, no collisions) and the capacitive discharge (walls, MCC),
          in each particle form, alone or several stepped as a group
  simnd   periodic 2D3V / 3D3V plasmas (SimulationND), uniform B
  walls   2D / 3D runs with field walls and reflecting or absorbing particle walls
  swarm   electron swarms: run_swarm_benchmark (swarm_run) or requests to a server
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "aurora-pic_b200"))
import apic  # noqa: E402
from apic import workloads as W  # noqa: E402

PRECISION = {"fp64": apic.FP64, "fp32": apic.FP32, "fp32_storage": apic.FP32_STORAGE}


def listed():
    return [
        # the smallest call a user makes: a 1D1V instability deck of a few thousand
        # particles whose phase space is plotted every 20 steps (launches and latency count)
        {"name": "two_stream_small", "kind": "sim1d", "deck": "two_stream", "cells": 128, "particles": 8192,
         "form": "fp64", "runs": 1, "steps": 20, "phase_space": True},
        # Landau damping with a million particles on a small mesh (many particles a cell)
        {"name": "landau_1m", "kind": "sim1d", "deck": "landau", "cells": 64, "particles": 1 << 20,
         "form": "fp64", "runs": 1, "steps": 40},
        # the capacitive discharge of the benchmark, in its FP64 form ...
        {"name": "ccp_fp64", "kind": "sim1d", "deck": "ccp", "cells": 512, "particles": 262144,
         "form": "fp64", "runs": 1, "steps": 40},
        # ... and in its FP32 cell form
        {"name": "ccp_fp32", "kind": "sim1d", "deck": "ccp", "cells": 512, "particles": 262144,
         "form": "fp32", "runs": 1, "steps": 40},
        # a parameter scan: eight discharges stepped together
        {"name": "ccp_group_fp32", "kind": "sim1d", "deck": "ccp", "cells": 512, "particles": 262144,
         "form": "fp32", "runs": 8, "steps": 40},
        # a mid-size 2D deck in the bit-faithful form, a ragged particle count, oblong mesh
        {"name": "plasma2d_fp64", "kind": "simnd", "nx": 256, "ny": 128, "nz": 1, "particles": 1048613,
         "form": "fp64", "sort": 16, "items": 0, "steps": 32},
        # the benchmark's 2D deck: 512^2, 64 particles a cell of each species
        {"name": "plasma2d_fp32", "kind": "simnd", "nx": 512, "ny": 512, "nz": 1, "particles": 512 * 512 * 64,
         "form": "fp32", "sort": 8, "items": 4, "steps": 64},
        # a mid-size 3D deck in the bit-faithful form
        {"name": "plasma3d_fp64", "kind": "simnd", "nx": 64, "ny": 64, "nz": 64, "particles": 64 ** 3 * 16,
         "form": "fp64", "sort": 16, "items": 0, "steps": 32},
        # the benchmark's 3D deck: 256^3, 8 particles a cell of each species
        {"name": "plasma3d_fp32", "kind": "simnd", "nx": 256, "ny": 256, "nz": 256, "particles": 256 ** 3 * 8,
         "form": "fp32", "sort": 3, "items": 2, "steps": 96},
        # a 2D channel: periodic along x, biased walls along y
        {"name": "walls2d", "kind": "walls", "nx": 512, "ny": 513, "nz": 1, "particles": 2000003, "steps": 40},
        # a closed 3D box with grounded walls
        {"name": "walls3d", "kind": "walls", "nx": 129, "ny": 129, "nz": 129, "particles": 4194304, "steps": 40},
        # the swarm server with a handful of requests in flight
        {"name": "swarm_serve", "kind": "swarm", "how": "serve", "form": "fp32", "requests": 12,
         "particles": 100000, "population": "fixed", "steps": 400},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sim1d", "sim1d", "sim1d", "simnd", "simnd", "simnd", "walls", "swarm"])
    if kind == "sim1d":
        deck = rng.choice(["two_stream", "landau", "ccp", "ccp"])
        form = rng.choice(["fp64", "fp64", "fp32", "fp32_storage"])
        if deck == "ccp":
            return {"kind": kind, "deck": deck, "cells": _log(rng, 64, 1000), "particles": _log(rng, 20000, 400000),
                    "form": form, "runs": rng.choice([1, 1, 3, 8]), "steps": rng.randint(10, 40)}
        return {"kind": kind, "deck": deck, "cells": _log(rng, 32, 1024), "particles": _log(rng, 2000, 1 << 20),
                "form": form, "runs": rng.choice([1, 1, 4]), "steps": rng.randint(10, 40),
                "phase_space": rng.random() < 0.25}
    if kind == "simnd":
        form = rng.choice(["fp64", "fp32"])
        if rng.random() < 0.5:
            n = [2 ** rng.randint(5, 10), 2 ** rng.randint(5, 9), 1]
            ppc, sort = rng.uniform(4, 64), rng.choice([4, 8, 16])
        else:
            n = [2 ** rng.randint(4, 8), 2 ** rng.randint(4, 7), 2 ** rng.randint(4, 7)]
            ppc, sort = rng.uniform(2, 16), rng.choice([3, 8, 16])
        particles = min(int(ppc * n[0] * n[1] * n[2]) + rng.randint(0, 63), 1 << 25)
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "particles": particles, "form": form,
                "sort": sort, "items": rng.choice([0, 0, 1, 2, 4]), "steps": sort * rng.randint(1, 2)}
    if kind == "walls":
        if rng.random() < 0.6:
            lx, ly = 2 ** rng.randint(5, 9), 2 ** rng.randint(5, 9)
            which = rng.choice(["x", "y", "xy"])
            across = _log(rng, 33, 700)  # a power of two would be a periodic extent
            across += across & (across - 1) == 0
            n = [across if which == "x" else lx + 1 if which == "xy" else lx,
                 across if which == "y" else ly + 1 if which == "xy" else ly, 1]
        else:
            n = [2 ** rng.randint(4, 7) + 1 for _ in range(3)]
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "particles": _log(rng, 30000, 3000000),
                "steps": rng.randint(10, 40)}
    return {"kind": kind, "how": rng.choice(["run", "serve"]), "form": rng.choice(["fp64", "fp32", "fp32"]),
            "requests": rng.randint(1, 16), "particles": _log(rng, 5000, 200000),
            "population": rng.choice(["fixed", "fixed", "branching"]), "steps": 20 * rng.randint(8, 20)}


# ---- what a program sets up once ------------------------------------------------------

def _deck1d(case, seed):
    if case["deck"] == "two_stream":
        return W.two_stream(particles_per_beam=case["particles"], nx=case["cells"], seed=seed)
    if case["deck"] == "landau":
        return W.landau(particles=case["particles"], nx=case["cells"], seed=seed)
    cells = case["cells"]
    wl = W.ccp_helium(particles_per_cell=1, cells=cells, seed=seed)
    rng = np.random.default_rng(seed)
    n = case["particles"]  # any count, not only a multiple of the cells
    for s in wl.species:
        s.weight = s.weight * cells / n
        s.capacity = int(n * 1.5) + 4096
        s.x = rng.uniform(0.0, wl.length, n)
        s.v, s.vy, s.vz = (s.thermal * rng.standard_normal(n) for _ in range(3))
    return wl


def _is3d(case):
    return case["nz"] > 1


# The benchmark's periodic plasma decks: cell = Debye length at n0 = 1e16 m^-3,
# dt = 0.1 / omega_pe; 2D: Te 2 eV, Ti 0.03 eV, Bz = 0.01 T, the lowest mode of both
# axes perturbed by 1e-3; 3D: Te 1 eV, Ti 0.025 eV, Bx = 0.005 T, the lowest x mode.
def _plan(case, seed):
    three = _is3d(case)
    cells = (case["nx"], case["ny"]) + ((case["nz"],) if three else ())
    plan = W.plasma_plan(3 if three else 2, cells=cells, ppc=1, seed=2 * seed + 1)
    scale = float(np.prod(cells)) / case["particles"]
    plan.species = [(q, m, w * scale, case["particles"], vt, s) for (q, m, w, _, vt, s) in plan.species]
    return plan


# Normalized units: electrons and ions 100 times heavier, unit density, cell 0.5 Debye
# lengths, dt = 0.1; the ions of half the thermal energy
def _walls(case):
    three = _is3d(case)
    n = (case["nx"], case["ny"]) + ((case["nz"],) if three else ())
    # a power of two is a periodic extent, everything else has walls
    wall = [bool(k & (k - 1)) for k in n]
    length = [0.5 * (k - 1 if w else k) for k, w in zip(n, wall)]
    weight = float(np.prod(length)) / case["particles"]
    species = [(-1.0, 1.0, weight, 1.0), (1.0, 100.0, weight, 0.07)]
    # the lower side of every wall axis absorbs, the upper one reflects
    boundaries = [k for w in wall for k in ((1, 2) if w else (3, 3))]
    potentials = None if three else [0.0, 1.5 if wall[0] else 0.0, 0.0, 1.5 if wall[1] else 0.0]
    return n, wall, length, species, boundaries, potentials, (0.0, 0.0, 0.2)


def _walls_particles(case, seed):
    n, wall, length, species, *_ = _walls(case)
    out = []
    for k, (q, m, w, vt) in enumerate(species):
        g = torch.Generator().manual_seed(1000003 * seed + k)
        np_ = case["particles"]
        pos = torch.rand((3, np_), generator=g, dtype=torch.float64)
        for a in range(3):
            pos[a] *= length[a] if a < len(n) else 0.0
        out.append((pos, vt * torch.randn((3, np_), generator=g, dtype=torch.float64)))
    return out


def prepare(case, seed):
    if case["kind"] == "sim1d":
        sims = []
        for r in range(case["runs"]):
            wl = _deck1d(case, 64 * seed + r)
            cfg, tables = W.to_device_config(wl, precision=PRECISION[case["form"]], seed=9000 + 64 * seed + r)
            sim = apic.Simulation1D(cfg, tables)
            for i, s in enumerate(wl.species):
                sim.load(i, s.x, s.v, None, s.vy, s.vz)
            sim.initialize()
            sims.append(sim)
        return {"case": case, "sims": sims}
    if case["kind"] == "simnd":
        plan = _plan(case, seed)
        sim = apic.SimulationND(plan.config(precision=PRECISION[case["form"]], sort_interval=case["sort"],
                                            push_items=case["items"]))
        plan.load(sim)
        sim.initialize()
        return {"case": case, "sim": sim}
    if case["kind"] == "walls":
        n, wall, length, species, boundaries, potentials, B = _walls(case)
        cfg = apic.config_nd(dims=len(n), n=n, length=length, dt=0.1, magnetic_field=B,
                             species=[(q, m, w, case["particles"]) for q, m, w, _ in species],
                             walls=(wall, potentials, boundaries))
        sim = apic.SimulationND(cfg)
        for k, (pos, v) in enumerate(_walls_particles(case, seed)):
            sim.load(k, pos.numpy(), v.numpy())
        sim.initialize()
        return {"case": case, "sim": sim}
    spec = W.swarm_c5(particles=case["particles"], steps=case["steps"], burn_in_steps=case["steps"] // 2,
                      seed=100 * seed + 1, branching=case["population"] == "branching")
    fields = [float(f) for f in np.geomspace(20.0, 600.0, case["requests"])]
    cfg, gas, tables = W.to_device_swarm(spec, precision=PRECISION[case["form"]])
    cfg.work_item_limit = 1 << 40
    state = {"case": case, "spec": spec, "fields": fields, "cfg": cfg, "gas": gas, "tables": tables}
    if case["how"] == "serve":
        state["server"] = apic.SwarmServer(gas, 4 << 30, max_runs=16, precision=PRECISION[case["form"]],
                                           steps_per_launch=100)
    return state


# ---- one pass -------------------------------------------------------------------------

def _result(r):
    if r.status != 0:
        raise RuntimeError(r.message.decode())
    return [r.mean_velocity_x, r.drift_velocity, r.mean_energy_ev, r.diffusion_longitudinal, r.diffusion_transverse,
            r.final_weight, r.ionization_rate, r.net_rate], [r.steps_done, r.final_particles, r.candidates,
                                                             r.null_collisions] + list(r.channel_collisions)


def run(state):
    case = state["case"]
    if case["kind"] == "sim1d":
        sims = state["sims"]
        if len(sims) == 1:
            sims[0].step(case["steps"])
        else:
            apic.step_group(sims, case["steps"])
        out = {"fields": [s.fields() for s in sims]}
        if case.get("phase_space"):
            out["particles"] = [[(p["x"], p["v"]) for p in map(s.particles, range(s.cfg.nspecies))] for s in sims]
        if case["deck"] == "ccp":
            counts = []
            for s in sims:
                t = s.collision_totals()
                counts += [t.candidates, t.null_collisions] + [c for m in t.channel_collisions for c in m]
                for k in range(2):
                    b = s.boundary_losses(k)
                    counts += [b.absorbed_left, b.absorbed_right, s.count(k)]
            out["counts"] = np.array(counts, dtype=np.int64)
        return out
    if case["kind"] in ("simnd", "walls"):
        sim = state["sim"]
        sim.step(case["steps"])
        out = {"fields": sim.fields()}
        if case["kind"] == "walls":
            out["counts"] = np.concatenate([sim.boundary_losses(k).astype(np.int64) for k in range(2)])
        return out
    if case["how"] == "run":
        results = apic.swarm_run(state["cfg"], state["gas"], state["fields"])
    else:
        srv, spec = state["server"], state["spec"]
        ids = [srv.submit(W.swarm_request(spec, f, seed=spec.seed + k)) for k, f in enumerate(state["fields"])]
        while True:
            active, queued = srv.advance()
            if not active and not queued:
                break
        results = [srv.poll(i) for i in ids]
    parts = [_result(r) for r in results]
    return {"values": np.array([p[0] for p in parts]), "counts": np.array([p[1] for p in parts], dtype=np.int64)}


# ---- what a pass cannot do without ------------------------------------------------------

def work(case):
    """The persistent state of every particle read and written once a step, the mesh's
    charge, potential and field written and read once a step, the fields returned."""
    kind = case["kind"]
    wide = case.get("form", "fp64") == "fp64"
    if kind == "sim1d":
        vdim = 3 if case["deck"] == "ccp" else 1
        state = 8 + 8 * vdim if wide else 8 + 4 * vdim
        if case["form"] == "fp32_storage":
            state = 8 + 4 * vdim
        n = case["particles"] * (1 if case["deck"] == "landau" else 2) * case["runs"]
        mesh = 8 * 3 * (case["cells"] + 1) * case["runs"]
        flops = 40 if vdim == 1 else 60
    elif kind == "simnd":
        three = _is3d(case)
        state = (48 if three else 40) if wide else (28 if three else 24)
        n, N = 2 * case["particles"], case["nx"] * case["ny"] * case["nz"]
        mesh = 8 * N * (5 if three else 4)
        flops = 170 if three else 100
    elif kind == "walls":
        three = _is3d(case)
        state = 48 if three else 40
        n, N = 2 * case["particles"], case["nx"] * case["ny"] * case["nz"]
        mesh = 8 * N * (5 if three else 4)
        flops = 170 if three else 100
    else:
        n, state, mesh, flops = case["particles"] * case["requests"], 48 if wide else 24, 0, 60
    steps = case["steps"]
    read = 16 * n if case.get("phase_space") else 0
    return {"bytes": float(steps * (2 * n * state + 2 * mesh) + mesh + read), "flops": float(steps * n * flops)}


# ---- the same pass in 64 bits, in plain torch -------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _philox(i, c2, seed):
    """Philox4x32-10 of counters (i, 0x5eed, c2, 0) under a 64-bit seed, as int64 words."""
    mask = 0xFFFFFFFF
    c = [i & mask, torch.full_like(i, 0x5EED), torch.full_like(i, c2), torch.zeros_like(i)]
    k0, k1 = seed & mask, (seed >> 32) & mask
    for r in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57  # 64-bit products, wrapped
        h0, h1 = (p0 >> 32) & mask, (p1 >> 32) & mask
        c = [h1 ^ c[1] ^ k0, p1 & mask, h0 ^ c[3] ^ k1, p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c


def _maxwellian(n, seed, lengths, vt, axis, amplitude, dev):
    """What SimulationND.load_maxwellian puts into the run: uniform positions displaced
    along the perturbed axes, normal velocities by Box and Muller."""
    dims = len(lengths)
    pos, vel = (torch.empty((k, n), dtype=torch.float64, device=dev) for k in (dims, 3))
    for lo in range(0, n, 1 << 24):
        i = torch.arange(lo, min(n, lo + (1 << 24)), dtype=torch.int64, device=dev)
        at = slice(lo, lo + len(i))

        def u(a, b):
            return (((a << 21) ^ (b & 0x1FFFFF)).double() + 0.5) * 2.0 ** -53

        r, r2 = _philox(i, 0, seed), _philox(i, 1, seed)
        for a, w in enumerate([u(r[0], r[1]), u(r[2], r[3]), u(r2[0], r2[1])][:dims]):
            x = w * lengths[a]
            if amplitude != 0.0 and (axis < 0 or axis == a):
                k = 2.0 * math.pi / lengths[a]
                x = torch.remainder(x + amplitude / k * torch.sin(k * x), lengths[a])
            pos[a, at] = x
        g, g2 = _philox(i, 2, seed), _philox(i, 3, seed)
        s1, s2 = (torch.sqrt(-2.0 * torch.log(u(h[0], h[1]))) for h in (g, g2))
        t1, t2 = (2.0 * math.pi * u(h[2], h[3]) for h in (g, g2))
        vel[0, at], vel[1, at], vel[2, at] = vt * s1 * torch.cos(t1), vt * s1 * torch.sin(t1), vt * s2 * torch.cos(t2)
    return pos, vel


class _Plain:
    """An electrostatic run in plain torch: linear shapes, leapfrog or Boris, periodic
    axes by FFT, wall axes by sine transforms.  Axis 0 is the fastest of the mesh."""

    def __init__(self, n, wall, length, eps, dt, species, B, potentials, spectral, dev):
        self.n, self.wall, self.L, self.eps, self.dt, self.dev = n, wall, length, eps, dt, dev
        self.d = [l / (k - 1 if w else k) for l, k, w in zip(length, n, wall)]
        self.species, self.B, self.pot, self.spectral = species, B, potentials, spectral
        self.losses = torch.zeros((len(species), 2 * len(n)), dtype=torch.int64, device=dev)
        self.solve()

    def stencil(self, pos):
        idx, wt = None, None
        stride = 1
        for a, n in enumerate(self.n):
            g = pos[a] / self.d[a]
            i = torch.floor(g)
            if self.wall[a]:
                i = i.clamp(0, n - 2)
            f = g - i
            i = i.long()
            j = [i, i + 1] if self.wall[a] else [i % n, (i + 1) % n]
            w = [1.0 - f, f]
            if idx is None:
                idx, wt = [k * stride for k in j], w
            else:
                idx, wt = [p + k * stride for k in j for p in idx], [p * q for q in w for p in wt]
            stride *= n
        return idx, wt

    def shape(self):
        return tuple(reversed(self.n))

    def chunks(self, s):
        n = s["pos"].shape[1]
        for lo in range(0, n, 1 << 24):
            yield slice(lo, min(n, lo + (1 << 24)))

    def solve(self):
        dims, dev = len(self.n), self.dev
        N = int(np.prod(self.n))
        rho = torch.zeros(N, dtype=torch.float64, device=dev)
        for s in self.species:
            # grid shares first, one scale for all of them (the shares stay of order one)
            share = torch.zeros(N, dtype=torch.float64, device=dev)
            for at in self.chunks(s):
                for i, w in zip(*self.stencil(s["pos"][:, at])):
                    share.index_add_(0, i, w)
            rho += share * (s["q"] * s["w"])
        rho = rho.reshape(self.shape())
        for a in range(dims):
            width = torch.full((self.n[a],), self.d[a], dtype=torch.float64, device=dev)
            if self.wall[a]:
                width[0] = width[-1] = 0.5 * self.d[a]
            rho = rho / width.reshape([-1 if dims - 1 - b == a else 1 for b in range(dims)])
        self.rho = rho
        hat, eig, inner = (rho - (rho.mean() if not any(self.wall) else 0.0)) / self.eps, 0.0, []
        phi = torch.zeros_like(rho)
        if any(self.wall):
            for a in range(dims):  # wall potentials
                if self.wall[a] and self.pot is not None:
                    ax = dims - 1 - a
                    phi.select(ax, 0).fill_(self.pot[2 * a])
                    phi.select(ax, -1).fill_(self.pot[2 * a + 1])
            if dims == 2 and all(self.wall) and self.pot is not None:
                l, r, b, t = self.pot
                phi[0, 0], phi[0, -1], phi[-1, 0], phi[-1, -1] = (l + b) / 2, (r + b) / 2, (l + t) / 2, (r + t) / 2
            for a in range(dims):
                ax = dims - 1 - a
                if self.wall[a]:
                    hat = hat.clone()
                    hat.select(ax, 1).add_(phi.select(ax, 0) / self.d[a] ** 2)
                    hat.select(ax, -2).add_(phi.select(ax, -1) / self.d[a] ** 2)
            for a in range(dims):
                if self.wall[a]:
                    inner.append(dims - 1 - a)
                    hat = hat.narrow(dims - 1 - a, 1, self.n[a] - 2)
        waves = []
        for a in range(dims):
            ax, n = dims - 1 - a, self.n[a]
            view = [-1 if b == ax else 1 for b in range(dims)]
            if self.wall[a]:
                m = n - 2
                k = torch.arange(1, m + 1, dtype=torch.float64, device=dev)
                S = torch.sin(math.pi / (m + 1) * torch.outer(k, k)) * math.sqrt(2.0 / (m + 1))
                hat = torch.movedim(torch.movedim(hat, ax, -1) @ S.to(hat.dtype), -1, ax)
                eig = eig + (4.0 * torch.sin(0.5 * math.pi * k / (m + 1)) ** 2 / self.d[a] ** 2).reshape(view)
                waves.append(S)
            else:
                hat = torch.fft.fft(hat, dim=ax)
                m = torch.arange(n, dtype=torch.float64, device=dev)
                m = torch.where(m <= n // 2, m, m - n)
                if self.spectral:
                    waves.append((2.0 * math.pi * m / self.L[a]).reshape(view))
                    eig = eig + waves[-1] ** 2
                else:
                    waves.append(None)
                    eig = eig + (4.0 * torch.sin(math.pi * m / n) ** 2 / self.d[a] ** 2).reshape(view)
        if not any(self.wall):
            origin = (0,) * dims
            eig[origin] = 1.0
            hat = hat / eig
            hat[origin] = 0.0
            self.phi = torch.fft.ifftn(hat).real
            self.E = torch.stack([torch.fft.ifftn(-1j * waves[a] * hat).real.reshape(-1) for a in range(dims)], -1)
            return
        hat = hat / eig
        for a in range(dims):
            ax = dims - 1 - a
            if self.wall[a]:
                hat = torch.movedim(torch.movedim(hat, ax, -1) @ waves[a].to(hat.dtype), -1, ax)
            else:
                hat = torch.fft.ifft(hat, dim=ax)
        hat = hat.real if hat.is_complex() else hat
        view = phi
        for ax in inner:
            view = view.narrow(ax, 1, phi.shape[ax] - 2)
        view.copy_(hat)
        self.phi = phi
        E = []
        for a in range(dims):
            ax = dims - 1 - a
            if self.wall[a]:
                e = torch.empty_like(phi)
                n = self.n[a]
                e.narrow(ax, 1, n - 2).copy_(-(phi.narrow(ax, 2, n - 2) - phi.narrow(ax, 0, n - 2)) / (2 * self.d[a]))
                e.select(ax, 0).copy_(-(phi.select(ax, 1) - phi.select(ax, 0)) / self.d[a])
                e.select(ax, -1).copy_(-(phi.select(ax, -1) - phi.select(ax, -2)) / self.d[a])
            else:
                e = -(torch.roll(phi, -1, ax) - torch.roll(phi, 1, ax)) / (2 * self.d[a])
            E.append(e.reshape(-1))
        self.E = torch.stack(E, -1)

    def kick(self, s, at, dt):
        idx, wt = self.stencil(s["pos"][:, at])
        e = 0.0
        for i, w in zip(idx, wt):
            e = e + self.E[i] * w[:, None]
        v = s["v"][:, at]
        h = 0.5 * s["q"] / s["m"] * dt
        dims = len(self.n)
        if self.B is None:
            for a in range(min(dims, v.shape[0])):
                v[a] += 2.0 * h * e[:, a]
            return
        t = [h * b for b in self.B]
        f = 2.0 / (1.0 + sum(b * b for b in t))
        u = [v[a] + h * e[:, a] if a < dims else v[a].clone() for a in range(3)]
        p = [u[0] + u[1] * t[2] - u[2] * t[1], u[1] + u[2] * t[0] - u[0] * t[2], u[2] + u[0] * t[1] - u[1] * t[0]]
        q = [u[0] + f * (p[1] * t[2] - p[2] * t[1]), u[1] + f * (p[2] * t[0] - p[0] * t[2]),
             u[2] + f * (p[0] * t[1] - p[1] * t[0])]
        for a in range(3):
            v[a] = q[a] + h * e[:, a] if a < dims else q[a]

    def start(self):
        for s in self.species:
            for at in self.chunks(s):
                self.kick(s, at, -0.5 * self.dt)

    def step(self, boundaries):
        for k, s in enumerate(self.species):
            gone = None
            for at in self.chunks(s):
                self.kick(s, at, self.dt)
                pos, v = s["pos"][:, at], s["v"][:, at]
                for a, L in enumerate(self.L):
                    x = pos[a] + v[a] * self.dt
                    if not self.wall[a]:
                        x = torch.where((x < 0) | (x >= L), torch.remainder(x, L), x)
                    pos[a] = x
            for side, kind in enumerate(boundaries or []):
                a, x, v = side >> 1, s["pos"][side >> 1], s["v"][side >> 1]
                out = x < 0.0 if side % 2 == 0 else x > self.L[a]
                if gone is not None:
                    out = out & ~gone
                if kind == 1:
                    self.losses[k, side] += out.sum()
                    gone = out if gone is None else gone | out
                elif kind == 2:
                    x.copy_(torch.where(out, -x if side % 2 == 0 else 2.0 * self.L[a] - x, x))
                    v.copy_(torch.where(out, -v, v))
            if gone is not None:
                s["pos"], s["v"] = s["pos"][:, ~gone], s["v"][:, ~gone]
        self.solve()

    def fields(self):
        N = int(np.prod(self.n))
        E = self.E.t().contiguous()
        return self.rho.reshape(-1), self.phi.reshape(-1), E[0] if len(self.n) == 1 else E.reshape(-1, N)


def _exact_1d(case, seed, r, dev):
    wl = _deck1d(case, 64 * seed + r)
    species = [{"q": s.charge, "m": s.mass, "w": s.weight,
                "pos": torch.from_numpy(s.x.copy()).to(dev)[None], "v": torch.from_numpy(s.v.copy()).to(dev)[None]}
               for s in wl.species]
    sim = _Plain((wl.nx,), (False,), (wl.length,), 1.0, wl.dt, species, None, None, True, dev)
    sim.start()
    for _ in range(case["steps"]):
        sim.step(None)
    out = sim.fields()
    if not case.get("phase_space"):
        return out, None
    particles = []
    for s in species:
        half = s["v"].clone()
        sim.kick(s, slice(None), 0.5 * wl.dt)  # time-centred velocity
        particles.append((s["pos"][0], s["v"][0]))
        s["v"] = half
    return out, particles


def exact(case, seed):
    """None where random collisions decide (discharges, swarms): their streams are the
    framework's own."""
    dev = _device()
    if case["kind"] == "sim1d" and case["deck"] != "ccp":
        runs = [_exact_1d(case, seed, r, dev) for r in range(case["runs"])]
        out = {"fields": [f for f, _ in runs]}
        if case.get("phase_space"):
            out["particles"] = [p for _, p in runs]
        return out
    if case["kind"] == "simnd":
        if case["particles"] * case["steps"] > 1.3e10:
            return None
        plan = _plan(case, seed)
        species = []
        for k, (q, m, w, n, vt, s) in enumerate(plan.species):
            pos, v = _maxwellian(n, s, plan.length, vt, plan.perturb_axis, plan.amplitude if k == 0 else 0.0, dev)
            species.append({"q": q, "m": m, "w": w, "pos": pos, "v": v})
        dims = len(plan.n)
        sim = _Plain(plan.n, (False,) * dims, plan.length, 8.8541878128e-12, plan.dt, species, plan.B, None, True, dev)
        sim.start()
        for _ in range(case["steps"]):
            sim.step(None)
        return {"fields": sim.fields()}
    if case["kind"] == "walls":
        n, wall, length, decks, boundaries, potentials, B = _walls(case)
        species = [{"q": q, "m": m, "w": w, "pos": pos[:len(n)].to(dev), "v": v.to(dev)}
                   for (q, m, w, _), (pos, v) in zip(decks, _walls_particles(case, seed))]
        sim = _Plain(n, wall, length, 1.0, 0.1, species, B, potentials, False, dev)
        sim.start()
        for _ in range(case["steps"]):
            sim.step(boundaries)
        return {"fields": sim.fields(), "counts": None}
    return None
