"""The workloads that the solver's speed is measured on, through its public Python binding.

A case is one call (or one short sequence of calls) as a user's program makes
it, on state that such a program keeps: lattices, decomposed domains,
ensembles, the solve server, and the diagnostics of a long run.  All of them
are lid-driven cavities in lattice units with a seeded start-up velocity.

Kinds of case
  lattice  one cavity stepped through Lattice.run, velocity and density kept
           (the binding's defaults), then both read back
  domain   a decomposed (or single) domain stepped through Domain.run with
           graph replay, velocity written on the last step and read back
  batch    an ensemble of uneven cavities: reset, run to completion, every
           velocity field read back
  server   requests submitted together, ticked until all have completed,
           every velocity field read back, the solves released
  monitor  the diagnostics that a precision study takes between runs: the
           conserved sums of a lattice and of its FP64 twin, and the velocity
           error of the one against the other
"""
import math

import numpy as np
import torch

from turbulent_lbm_multigpu_gb300 import capi

BYTES = {"f32": 4, "f64": 8, "f16": 2, "bf16": 2, "c16": 2}
# Arithmetic of one cell update: moments 45, density and |u|^2 7, equilibria 85, relaxation 57; subgrid model 81 more.
FLOPS_BGK, FLOPS_LES = 194, 81
AMP = 1e-3  # start-up velocity amplitude
QUANTUM = 64  # steps per server tick


def listed():
    return [
        # the smallest call: two steps of a tiny cavity and a look at its fields (interactive use, tests, coupling)
        {"name": "lattice 24x20x16 f32, 2 steps", "kind": "lattice", "nx": 24, "ny": 20, "nz": 16, "storage": "f32",
         "steps": 2, "re": 1000.0, "lid": 0.05, "cs": 0.17},
        # the classic validation cavity, fields kept
        {"name": "lattice 64^3 f32, 99 steps", "kind": "lattice", "nx": 64, "ny": 64, "nz": 64, "storage": "f32",
         "steps": 99, "re": 1000.0, "lid": 0.05, "cs": 0.17},
        # odd extents in half storage: rows that are not whole 16-byte units
        {"name": "lattice 121x99x87 f16, 50 steps", "kind": "lattice", "nx": 121, "ny": 99, "nz": 87, "storage": "f16",
         "steps": 50, "re": 5000.0, "lid": 0.1, "cs": 0.17},
        # the headline workload: a decomposed domain with its halo exchange, in float ...
        {"name": "domain 256^3 2x2x1 f32, 20 steps", "kind": "domain", "nx": 256, "ny": 256, "nz": 256, "px": 2, "py": 2,
         "pz": 1, "storage": "f32", "steps": 20, "re": 10000.0, "lid": 0.1, "cs": 0.17, "fma64": False},
        # ... and in double, with the reference arithmetic
        {"name": "domain 256^3 2x2x1 f64, 8 steps", "kind": "domain", "nx": 256, "ny": 256, "nz": 256, "px": 2, "py": 2,
         "pz": 1, "storage": "f64", "steps": 8, "re": 10000.0, "lid": 0.1, "cs": 0.17, "fma64": False},
        # double with fused multiply-adds, smaller, the production setting where bits need not match the reference
        {"name": "domain 160x128x96 f64 fma, 20 steps", "kind": "domain", "nx": 160, "ny": 128, "nz": 96, "px": 2, "py": 1,
         "pz": 1, "storage": "f64", "steps": 20, "re": 10000.0, "lid": 0.1, "cs": 0.17, "fma64": True},
        # the largest float lattice of the bandwidth target
        {"name": "domain 512^3 f32, 20 steps", "kind": "domain", "nx": 512, "ny": 512, "nz": 512, "px": 1, "py": 1,
         "pz": 1, "storage": "f32", "steps": 20, "re": 10000.0, "lid": 0.1, "cs": 0.17, "fma64": False},
        # long turbulent runs in 16 bits: half storage ...
        {"name": "domain 384^3 f16, 20 steps", "kind": "domain", "nx": 384, "ny": 384, "nz": 384, "px": 1, "py": 1,
         "pz": 1, "storage": "f16", "steps": 20, "re": 20000.0, "lid": 0.1, "cs": 0.17, "fma64": False},
        # ... and the 13-bit significand where half is too coarse, decomposed
        {"name": "domain 256^3 2x2x1 c16, 20 steps", "kind": "domain", "nx": 256, "ny": 256, "nz": 256, "px": 2, "py": 2,
         "pz": 1, "storage": "c16", "steps": 20, "re": 20000.0, "lid": 0.1, "cs": 0.17, "fma64": False},
        # an ensemble of uneven cavities (parameter study), float and half mixed
        {"name": "batch of 40 cavities", "kind": "batch", "count": 40, "lo": 32, "hi": 128, "steps_lo": 20,
         "steps_hi": 120, "specs": 42},
        # a burst of requests through the solve server
        {"name": "server, 16 requests", "kind": "server", "count": 16, "lo": 32, "hi": 160, "steps_lo": 30,
         "steps_hi": 300, "specs": 7},
        # diagnostics between the runs of a precision study
        {"name": "monitor 256^3 f16 against f64", "kind": "monitor", "nx": 256, "ny": 256, "nz": 256, "storage": "f16",
         "re": 20000.0, "lid": 0.1, "cs": 0.17},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lattice", "lattice", "domain", "domain", "domain", "batch", "server", "monitor"])
    c = {"kind": kind}
    if kind in ("batch", "server"):
        c.update(count=_log(rng, 4, 40 if kind == "batch" else 16), lo=32, hi=128 if kind == "batch" else 160,
                 steps_lo=20, steps_hi=rng.randint(60, 120) if kind == "batch" else rng.randint(100, 300),
                 specs=rng.randrange(1 << 20))
        return c
    c.update(re=float(rng.randint(100, 20000)), lid=round(rng.uniform(0.02, 0.1), 3), cs=rng.choice([0.17, 0.17, 0.0]))
    if kind == "lattice":
        c.update(nx=_log(rng, 16, 144), ny=_log(rng, 16, 144), nz=_log(rng, 16, 144),
                 storage=rng.choice(["f32", "f16", "bf16", "c16", "f64"]), steps=_log(rng, 2, 100))
    elif kind == "monitor":
        c.update(nx=_log(rng, 48, 256), ny=_log(rng, 48, 256), nz=_log(rng, 48, 256),
                 storage=rng.choice(["f32", "f16", "bf16", "c16"]))
    else:
        storage = rng.choice(["f32", "f32", "f16", "c16", "f64"])
        hi = 256 if storage == "f64" else 400
        px, py, pz = rng.choice([(1, 1, 1), (2, 2, 1), (2, 1, 1), (1, 2, 2), (2, 2, 2)])
        c.update(nx=px * _log(rng, 32, hi // px), ny=py * _log(rng, 32, hi // py), nz=pz * _log(rng, 32, hi // pz),
                 px=px, py=py, pz=pz, storage=storage, steps=rng.randint(4, 20) if storage != "f64" else rng.randint(2, 8),
                 fma64=storage == "f64" and rng.random() < 0.5)
    return c


# ------------------------------------------------------------- the cavities
def _tau(lid, length, re):
    return 3.0 * lid * length / re + 0.5


def _params(storage, tau, cs, lid):
    if storage == "f64":
        t, inv = float(tau), 1.0 / float(tau)
    else:
        t32 = np.float32(tau)
        t, inv = float(t32), float(np.float32(1) / t32)
    return capi.Params.make(inv, t, capi.les_coefficient(cs), (0.0, 0.0, 0.0), lid)


def _specs(case):
    """Sizes, parameters, storage and step counts of an ensemble's cavities (the start-up seed comes with prepare)."""
    r = np.random.default_rng(case["specs"])
    out = []
    for _ in range(case["count"]):
        dims = [int(v) for v in np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), 3)).round()]
        re, lid = float(r.uniform(100, 5000)), float(r.uniform(0.02, 0.1))
        steps = int(r.integers(case["steps_lo"], case["steps_hi"] + 1))
        out.append({"dims": dims, "tau": _tau(lid, dims[0], re), "cs": 0.17, "lid": lid, "steps": steps,
                    "storage": "f16" if r.random() < 0.5 else "f32"})
    return out


def _lattice(case, storage, seed, fields):
    dims = (case["nx"], case["ny"], case["nz"])
    L = capi.Lattice(*dims, capi.STORAGE_NAMES[storage], fields, fields)
    L.set_params(_params(storage, _tau(case["lid"], dims[0], case["re"]), case["cs"], case["lid"]))
    L.init([capi.FLAG_OBSTACLE] * 6)
    L.write(capi.FIELD_FLAGS, np.full((dims[2] - 2) * (dims[0] - 2), capi.FLAG_VELOCITY_INJECTION, np.int32),
            origin=(1, dims[1] - 2, 1), size=(dims[0] - 2, 1, dims[2] - 2))
    L.perturb((0, 0, 0), dims, seed, AMP)
    return L


def _host(planes, dims, storage):
    """A pinned host buffer for `planes` planes of a lattice."""
    t = torch.empty((planes, dims[2], dims[1], dims[0]), dtype=torch.float64 if storage == "f64" else torch.float32,
                    pin_memory=True)
    return t.numpy()


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "lattice":
        dims = (case["nx"], case["ny"], case["nz"])
        s.update(L=_lattice(case, case["storage"], seed, True), done=0, u=_host(3, dims, case["storage"]),
                 rho=_host(1, dims, case["storage"]))
    elif kind == "domain":
        D = capi.Domain((case["nx"], case["ny"], case["nz"]), (case["px"], case["py"], case["pz"]),
                        capi.STORAGE_NAMES[case["storage"]], store_velocity=True)
        if case["fma64"]:
            D.set_fp64_contraction(True)
        if case["px"] * case["py"] * case["pz"] > 1:
            D.set_halo_mode(1)
        D.set_store_interval(0)
        D.set_params(_params(case["storage"], _tau(case["lid"], case["nx"], case["re"]), case["cs"], case["lid"]))
        D.reset()
        D.perturb(seed, AMP)
        s.update(D=D, u=[_host(3, D.sub, case["storage"]) for _ in D.subdomains])
    elif kind in ("batch", "server"):
        specs = _specs(case)
        s["cavities"] = [capi.Cavity.make(c["dims"], capi.STORAGE_NAMES[c["storage"]], c["tau"], c["cs"], c["lid"],
                                          c["steps"], (seed * 1000003 + i) & 0xFFFFFFFF, AMP) for i, c in enumerate(specs)]
        s["u"] = [_host(3, c["dims"], c["storage"]) for c in specs]
        if kind == "batch":
            s["B"] = capi.Batch(s["cavities"], store_velocity=True)
            s["B"].set_kernel_shape(3)
        else:
            s["S"] = capi.Server(150e9, store_velocity=True)
    else:
        s.update(L=_lattice(case, case["storage"], seed, False), R=_lattice(case, "f64", seed, False))
        s["L"].run(0, 2)
        s["R"].run(0, 2)
    capi.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "lattice":
        L, steps = s["L"], s["case"]["steps"]
        L.run(s["done"], steps)
        s["done"] += steps
        return {"u": L.read(capi.FIELD_VELOCITY, out=s["u"]), "rho": L.read(capi.FIELD_DENSITY, out=s["rho"])}
    if kind == "domain":
        s["D"].run(s["case"]["steps"], use_graph=True)
        return [L.read(capi.FIELD_VELOCITY, out=u) for L, u in zip(s["D"].subdomains, s["u"])]
    if kind == "batch":
        B = s["B"]
        B.reset()
        B.run(use_graph=True)
        return [L.read(capi.FIELD_VELOCITY, out=u) for L, u in zip(B.lattices, s["u"])]
    if kind == "server":
        S = s["S"]
        at = {S.submit(c): i for i, c in enumerate(s["cavities"])}
        while at:
            S.tick(max_steps=QUANTUM)
            for sid in S.poll():
                S.lattice(sid).read(capi.FIELD_VELOCITY, out=s["u"][at.pop(sid)])
                S.release(sid)
        return s["u"]
    L, R = s["L"], s["R"]
    e = capi.compare_velocity(L, 1, R, 1)
    a, b = L.reduce_conserved(1), R.reduce_conserved(1)
    return {"mass": a[0], "momentum": a[1:4], "energy": a[4], "mass64": b[0], "momentum64": b[1:4], "energy64": b[4],
            "error": [e[k] for k in ("max_abs", "rms", "rel_rms", "rel_max", "ref_rms", "ref_max")], "cells": e["cells"]}


def work(case):
    kind = case["kind"]
    if kind in ("batch", "server"):
        each = [(c["dims"][0] * c["dims"][1] * c["dims"][2], c["storage"], c["steps"], 0.17) for c in _specs(case)]
    else:
        n = case["nx"] * case["ny"] * case["nz"]
        if kind == "monitor":  # both lattices read once (one pass could give the sums and the errors), flags once
            return {"bytes": n * (19 * (BYTES[case["storage"]] + 8) + 1.0), "flops": n * 150.0}
        each = [(n, case["storage"], case["steps"], case["cs"])]
    b = f = 0.0
    for n, storage, steps, cs in each:
        real = 8 if storage == "f64" else 4
        b += n * steps * (38.0 * BYTES[storage] + 1) + n * real * (4 if kind == "lattice" else 3)
        f += n * steps * float(FLOPS_BGK + (FLOPS_LES if cs else 0))
    return {"bytes": b, "flops": f}


# ------------------------------------------------- the model in 64 bits, in torch
E = np.array([[1, -1, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0, 0, 0, 0],
              [0, 0, 1, -1, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1, 0, 0, 0],
              [0, 0, 0, 0, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1, 1, -1, 0]], dtype=np.int64)
W = np.array([1 / 18] * 4 + [1 / 36] * 12 + [1 / 18] * 2 + [1 / 3])
OPP = [i ^ 1 if i < 18 else 18 for i in range(19)]


def _startup(dims, seed, amp):
    """Start-up velocity: uniform on [-amp, amp) per component inside the walls, Philox4x32-10 keyed by (seed, cell)."""
    nx, ny, nz = dims
    m = 0xFFFFFFFF
    c = [torch.arange(nx * ny * nz, dtype=torch.int64, device="cuda")] + [torch.zeros(1, dtype=torch.int64, device="cuda")] * 3
    c[1] = c[0] >> 32
    c[0] = c[0] & m
    k0, k1 = seed & m, (seed >> 32) & m
    for _ in range(10):
        hi, lo = [], []
        for mult, v in ((0xD2511F53, c[0]), (0xCD9E8D57, c[2])):
            low = mult * (v & 0xFFFF)  # 32 x 32 -> 64 bits in two steps below 2^63
            high = mult * (v >> 16) + (low >> 16)
            hi.append((high >> 16) & m)
            lo.append(((high << 16) | (low & 0xFFFF)) & m)
        c = [hi[1] ^ c[1] ^ k0, lo[1], hi[0] ^ c[3] ^ k1, lo[0]]
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    u = torch.stack([((v >> 8).double() / 16777216.0 * 2 - 1) * amp for v in c[:3]]).view(3, nz, ny, nx)
    inside = torch.zeros((nz, ny, nx), dtype=torch.float64, device="cuda")
    inside[1:-1, 1:-1, 1:-1] = 1
    return u * inside


def _simulate(dims, tau, cs, lid, seed, amp, steps):
    """Start-up velocity, the velocity that the last of `steps` steps leaves, and the populations after it."""
    nx, ny, nz = dims
    n = nx * ny * nz
    wall = torch.zeros((nz, ny, nx), dtype=torch.bool, device="cuda")
    wall[0] = wall[-1] = True
    wall[:, 0] = wall[:, -1] = True
    wall[:, :, 0] = wall[:, :, -1] = True
    moving = torch.zeros_like(wall)
    moving[1:-1, ny - 2, 1:-1] = True
    wi, mi = (b.reshape(-1).nonzero().squeeze(1) for b in (wall, moving))
    e = torch.from_numpy(E).cuda().double()
    w = torch.from_numpy(W).cuda()[:, None]

    def equilibrium(u, a):
        eu = e.T @ u
        return eu.mul(4.5).add_(3.0).mul_(eu).add_(a).mul_(w)

    u0 = _startup(dims, seed, amp)
    u = u0.view(3, n)
    f = equilibrium(u, 1.0 - 1.5 * (u * u).sum(0))
    ul = torch.zeros((3, 1), dtype=torch.float64, device="cuda")
    ul[0] = lid
    fl = equilibrium(ul, 1.0 - 1.5 * (ul * ul).sum(0))
    second = torch.stack([e[a] * e[b] for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))])
    g = torch.empty_like(f)
    for _ in range(steps):
        for i in range(19):
            ex, ey, ez = (int(v) for v in E[:, i])
            p = f[i].view(nz, ny, nx)
            axes = [(s, d) for s, d in ((ez, 0), (ey, 1), (ex, 2)) if s]
            g[i] = (torch.roll(p, [a[0] for a in axes], [a[1] for a in axes]) if axes else p).reshape(-1)
        rho, u = g.sum(0), e @ g
        om = 1.0 / tau
        if cs:
            pi = second @ g
            q = 0
            for k, (a, b) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
                t = pi[k] - u[a] * u[b] - (rho / 3 if a == b else 0)
                q = q + t * t * (1 if a == b else 2)
            om = 2.0 / (tau + torch.sqrt(tau * tau + 18 * math.sqrt(2.0) * cs * cs * torch.sqrt(q)))
        f = equilibrium(u, rho - 1.5 * (u * u).sum(0))
        f.sub_(g).mul_(om).add_(g)
        f[:, wi] = g[:, wi][OPP]
        f[:, mi] = fl
        u[:, wi] = 0
        u[:, mi] = ul
    return u0, u.view(3, nz, ny, nx), f


def exact(case, seed):
    kind = case["kind"]
    if case.get("storage") == "bf16":
        return None  # its 8-bit significand leaves too few digits of a start-up field to compare
    if kind in ("batch", "server"):
        return [_simulate(c["dims"], c["tau"], c["cs"], c["lid"], (seed * 1000003 + i) & 0xFFFFFFFF, AMP, c["steps"])[1]
                for i, c in enumerate(_specs(case))]
    dims = [case["nx"], case["ny"], case["nz"]]
    tau = _tau(case["lid"], dims[0], case["re"])
    if kind == "lattice":
        return {"u": _simulate(dims, tau, case["cs"], case["lid"], seed, AMP, case["steps"])[1], "rho": None}
    if kind == "domain":
        # the subdomains overlap by two cells: together they are one smaller domain, ghost cells keep the start-up velocity
        p = [case["px"], case["py"], case["pz"]]
        sub = [d // k for d, k in zip(dims, p)]
        whole = [k * (v - 2) + 2 for k, v in zip(p, sub)]
        u0, u, _ = _simulate(whole, tau, case["cs"], case["lid"], seed, AMP, case["steps"])
        out = []
        for i in range(p[0] * p[1] * p[2]):
            at = [i % p[0], i // p[0] % p[1], i // (p[0] * p[1])]
            cut = tuple(slice(a * (v - 2), a * (v - 2) + v) for a, v in zip(at, sub))[::-1]
            part = u[(slice(None),) + cut].clone()
            for axis in (0, 1, 2):
                for end, ghost in ((0, at[axis] > 0), (-1, at[axis] < p[axis] - 1)):
                    if ghost:
                        face = [slice(None)] * 4
                        face[3 - axis] = end
                        part[tuple(face)] = u0[(slice(None),) + cut][tuple(face)]
            out.append(part)
        return out
    f = _simulate(dims, tau, case["cs"], case["lid"], seed, AMP, 2)[2]
    fluid = torch.zeros((dims[2], dims[1], dims[0]), dtype=torch.bool, device="cuda")
    fluid[1:-1, 1:-1, 1:-1] = True
    fluid[:, dims[1] - 2] = False
    f = f[:, fluid.view(-1)]
    j = torch.from_numpy(E).cuda().double() @ f
    mass, mom, en = float(f.sum()), j.sum(1).cpu().numpy(), 0.5 * float((j * j).sum())
    return {"mass": mass, "momentum": mom, "energy": en, "mass64": mass, "momentum64": mom, "energy64": en,
            "error": None, "cells": None}
