"""The work that programs have this framework do, as cases that can be timed.

A case is a dict; its "what" names the way in:

  frame     a resident handle advances some substeps and hands its bodies on: FP32-mixed runs
            as the float records of a renderer or engine in a device buffer, FP64 runs as the
            Body array in the program's pinned buffer
  ensemble  the same for many independent galaxies in one handle
  quasar    cosmosim_step of a quasar-mode handle (jets, accretion, lobes), then the records
  step      integrator_step on the caller's Body array and node pool, as the reference's main
            loop calls it (pageable or pinned memory)
  passes    the free functions one by one on host arrays: octree_build, octree_compute_forces,
            sph_compute_density, sph_compute_forces, sph_apply_cooling
  diagnose  a run's accuracy checks: FP64 direct sum on a sample, total energy
  adjoint   loss and gradient of a leapfrog run (csg_adjoint_forward, csg_adjoint_backward)

Bodies come from csg_generate_ics: 0 exponential disk, 1 two-disk merger with 10% SPH gas,
2 Plummer bulge + disk, 3 ensemble galaxy, 4 merger of stars. Every state keeps evolving from
pass to pass, as a simulation does.
"""
import math

import numpy as np
import torch
import torch.utils.checkpoint

from cosmosim_gb300 import lib
from cosmosim_gb300.abi import BODY_DTYPE, NODE_DTYPE, ptr

PREC = {"fp32": lib.PREC_FP32_MIXED, "fp64": lib.PREC_FP64}
STEP_FIELDS = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az")
SPH_FIELDS = ("density", "pressure", "internal_energy", "smoothing_h")
SAMPLE = 4096  # bodies of a direct-sum check
GAS_MIN_U, COOL, GAMMA, MAX_NB = 0.01, 0.05, 5.0 / 3.0, 128


def listed():
    return [
        # smallest interactive scene: every frame is launches and latency
        dict(name="frame_disk2k_fp32", what="frame", kind=0, n=2000, theta=0.5, eps=0.01, dt=1e-3,
             sph=False, prec="fp32", substeps=1, out="render"),
        # the reference's default run: 20,000 bodies, 8 FP64 substeps per frame
        dict(name="frame_disk20k_fp64", what="frame", kind=0, n=20000, theta=0.5, eps=0.01,
             dt=1e-3, sph=False, prec="fp64", substeps=8, out="bodies"),
        # quasar mode as an engine plugin drives it, one step (two substeps) a frame
        dict(name="quasar_20k_fp64", what="quasar", n=20000, merger=False),
        # the 100k merger with SPH, FP32-mixed, several substeps per displayed frame
        dict(name="frame_merger100k_fp32", what="frame", kind=1, n=100000, theta=0.5, eps=0.01,
             dt=1e-3, sph=True, prec="fp32", substeps=4, out="ue"),
        # the same system as a production FP64 run that writes its bodies out
        dict(name="frame_merger100k_fp64", what="frame", kind=1, n=100000, theta=0.5, eps=0.01,
             dt=1e-3, sph=True, prec="fp64", substeps=2, out="bodies"),
        # large-N: a million bodies, FP32-mixed and FP64
        dict(name="frame_bulge1m_fp32", what="frame", kind=2, n=1000000, theta=0.5, eps=0.005,
             dt=1e-3, sph=False, prec="fp32", substeps=1, out="render"),
        dict(name="frame_bulge1m_fp64", what="frame", kind=2, n=1000000, theta=0.5, eps=0.005,
             dt=1e-3, sph=False, prec="fp64", substeps=1, out="bodies"),
        # a parameter study: 64 galaxies of 2k to 50k bodies in one handle
        dict(name="ensemble64_fp32", what="ensemble", systems=64, n_min=2000, n_max=50000,
             size_seed=12, theta=0.5, eps=0.01, dt=1e-3, prec="fp32", substeps=1),
        # drop-in callers: the main loop's call on malloc'ed arrays, an odd body count
        dict(name="step_merger30001_fp64", what="step", kind=1, n=30001, theta=0.5, eps=0.01,
             dt=1e-3, sph=True, pinned=False),
        # the free functions one by one, as the reference's test program calls them
        dict(name="passes_merger5003", what="passes", kind=1, n=5003, theta=0.5, eps=0.01,
             dt=1e-3),
        # the checks of a production run: direct sum on 4096 bodies, energy over all pairs
        dict(name="diagnose_merger100k", what="diagnose", kind=1, n=100000, eps=0.01),
        # gradient of a short 10k-star merger run (one checkpoint segment)
        dict(name="adjoint10k", what="adjoint", n=10000, theta=0.5, eps=0.01, dt=2e-3, substeps=20,
             checkpoint=20),
    ]


def draw(rng):
    """One more case: the ways in by how often programs use them, sizes log-uniform."""
    size = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    theta = round(rng.uniform(0.3, 0.7), 3)
    what = rng.choice(["frame"] * 6 + ["ensemble", "quasar", "step", "step", "passes", "diagnose",
                                       "adjoint"])
    if what == "frame":
        kind, prec = rng.choice([0, 1, 2, 2]), rng.choice(["fp32", "fp64"])
        sph = kind == 1 and rng.random() < 0.7
        n = size(2000, 150000 if sph else 1000000)
        k = rng.choice([1, 2, 4])
        while k > 1 and k * n * _interactions(n, theta) > 2e8:
            k //= 2
        while n * _interactions(n, theta) > 2e9:
            theta = round(theta + 0.05, 3)
        out = "bodies" if prec == "fp64" else rng.choice(["render", "ue"])
        return dict(what=what, kind=kind, n=n, theta=theta, eps=rng.choice([0.005, 0.01, 0.02]),
                    dt=1e-3, sph=sph, prec=prec, substeps=k, out=out)
    if what == "ensemble":
        hi = size(2000, 50000)
        return dict(what=what, systems=rng.randint(3, 48), n_min=max(200, hi // 25), n_max=hi,
                    size_seed=rng.randint(1, 10 ** 6), theta=max(theta, 0.4), eps=0.01, dt=1e-3,
                    prec=rng.choice(["fp32", "fp32", "fp64"]), substeps=1)
    if what == "quasar":
        return dict(what=what, n=size(2000, 60000), merger=rng.random() < 0.5)
    if what == "step":
        return dict(what=what, kind=rng.choice([0, 1]), n=size(500, 120000), theta=theta, eps=0.01,
                    dt=1e-3, sph=rng.random() < 0.5, pinned=rng.random() < 0.5)
    if what == "passes":
        return dict(what=what, kind=1, n=size(500, 40000), theta=theta, eps=0.01, dt=1e-3)
    if what == "diagnose":
        return dict(what=what, kind=rng.choice([0, 1, 2]), n=size(5000, 100000), eps=0.01)
    t = rng.randint(4, 20)
    return dict(what=what, n=size(500, 12000), theta=max(theta, 0.4), eps=0.01, dt=2e-3, substeps=t,
                checkpoint=rng.randint(2, t))


def _interactions(n, theta):
    """Interactions per body of a Barnes-Hut walk, from this repository's measured counts
    (705 at 20k and 2129 at 1M, theta 0.5; 7536 at 1M, theta 0.3), fitted."""
    return min(float(n), 52.0 * (n / 1e3) ** 0.28 * theta ** -2.4 * 1.12)


def work(case):
    """Bytes and operations a pass cannot do without: the bodies' state read once and written
    once (plus what is handed on), 20 operations an interaction, and for SPH about 60 for each
    of up to 128 neighbours of the gas bodies in each of its two passes."""
    what = case["what"]
    if what == "ensemble":
        counts = _counts(case)
        flops = case["substeps"] * sum(20.0 * c * _interactions(c, case["theta"]) for c in counts)
        return {"bytes": sum(counts) * (10 * 8 + 9 * 8 + 40.0), "flops": flops}
    n = case["n"]
    if what == "diagnose":
        return {"bytes": n * 64.0 + min(SAMPLE, n) * 28.0,
                "flops": 20.0 * min(SAMPLE, n) * n + 12.0 * n * (n - 1) / 2}
    theta = case.get("theta", 0.5)
    inter = n * _interactions(n, theta)
    sph = case.get("sph", what in ("quasar", "passes"))
    gas = 0.1 * n * 128 * 60 * 2 if sph else 0.0
    if what == "adjoint":  # forward, and a backward of about 40 operations an interaction
        return {"bytes": n * (168.0 + 24 + 48), "flops": case["substeps"] * inter * (20 + 40.0)}
    if what in ("step", "passes"):  # Body records in and out, pool records (about 1.6 per body) out
        return {"bytes": n * (168.0 + 13 * 8 + 1.6 * 104), "flops": 20 * inter + gas}
    k = case.get("substeps", 2)
    out = {"render": 40.0, "ue": 64.0, "bodies": 168.0}[case.get("out", "ue")]
    return {"bytes": n * (14 * 8 + 13 * 8 + out), "flops": k * (20 * inter + gas)}


# ---- inputs ---------------------------------------------------------------------------------


def _counts(case):
    r = np.random.default_rng(case["size_seed"])
    u = r.uniform(math.log(case["n_min"]), math.log(case["n_max"]), case["systems"])
    return [int(v) for v in np.exp(u)]


def _ics_seed(seed):
    return 0x5EED0000 + 1000003 * (int(seed) % (1 << 40))


def _bodies(case, seed):
    if case["what"] == "ensemble":
        parts = [lib.generate_ics(3, c, _ics_seed(seed) + g) for g, c in enumerate(_counts(case))]
        out = np.zeros(sum(len(p) for p in parts), dtype=BODY_DTYPE)
        at = 0
        for p in parts:
            out[at:at + len(p)] = p
            at += len(p)
        return out
    return lib.generate_ics(case.get("kind", 4), case["n"], _ics_seed(seed))


def _sample(case, seed):
    r = np.random.default_rng(int(seed) + 1)
    k = min(SAMPLE, case["n"])
    return np.sort(r.choice(case["n"], size=k, replace=False)).astype(np.int32)


def _target(case, seed):
    """A target snapshot near the initial state (a program fits observed positions)."""
    b = _bodies(case, seed)
    r = np.random.default_rng(int(seed) + 2)
    x = np.stack([b["x"], b["y"], b["z"]], axis=1)
    v = np.stack([b["vx"], b["vy"], b["vz"]], axis=1)
    return x + v * case["dt"] * case["substeps"] + 0.05 * r.standard_normal(x.shape)


def _pinned(dtype, n):
    t = torch.empty(n * dtype.itemsize, dtype=torch.uint8, pin_memory=True)
    t.zero_()
    a = t.numpy().view(dtype)
    return t, a


def _turn(b, angle):
    """The system turned about z (positions, velocities, accelerations)."""
    c, s = math.cos(angle), math.sin(angle)
    for p, q in (("x", "y"), ("vx", "vy"), ("ax", "ay")):
        u, w = b[p].copy(), b[q].copy()
        b[p], b[q] = c * u - s * w, s * u + c * w


def prepare(case, seed):
    what = case["what"]
    st = {"case": case}
    if what == "quasar":
        cfg = lib.load().cosmosim_default_config()
        cfg.n_bodies, cfg.quasar, cfg.merger = case["n"], 1, int(case["merger"])
        sim = lib.Sim.from_config(cfg)
        b = sim.bodies()  # the library's own galaxy, turned: a scene that a program places
        _turn(b, 2 * math.pi * np.random.default_rng(int(seed)).random())
        sim.set_bodies(b)
        sim.sync()
        st["sim"] = sim
        st["rows"] = torch.zeros((case["n"] * 2, 16), dtype=torch.float32, device="cuda")
        return st
    b = _bodies(case, seed)
    if what in ("frame", "ensemble"):
        kw = dict(softening=case["eps"], theta=case["theta"], dt=case["dt"],
                  precision=PREC[case["prec"]], substeps=case["substeps"])
        if what == "ensemble":
            st["sim"] = lib.Sim.ensemble(b, _counts(case), **kw)
        else:
            st["sim"] = lib.Sim.from_bodies(b, sph=case["sph"], **kw)
        out = case.get("out", "render" if case["prec"] == "fp32" else "bodies")
        st["out"] = out
        if out == "bodies":
            st["keep"], st["host"] = _pinned(BODY_DTYPE, len(b))
        else:
            st["rows"] = torch.zeros((len(b), 16 if out == "ue" else 10), dtype=torch.float32,
                                     device="cuda")
    elif what == "step":
        if case["pinned"]:
            st["keep"], host = _pinned(BODY_DTYPE, len(b))
            host[:] = b
            st["keep2"], pool = _pinned(NODE_DTYPE, 8 * len(b))
        else:
            host, pool = b, np.zeros(8 * len(b), dtype=NODE_DTYPE)
        lib.integrator_init_accelerations(host, 1.0, case["eps"], case["theta"], pool)
        st["host"], st["pool"] = host, pool
    elif what == "passes":
        st["host"], st["pool"] = b, np.zeros(8 * len(b), dtype=NODE_DTYPE)
    elif what == "diagnose":
        st["sim"] = lib.Sim.from_bodies(b, softening=case["eps"])
        st["idx"] = _sample(case, seed)
    else:
        st["host"], st["target"] = b, _target(case, seed)
        st["adj"] = lib.Adjoint(len(b), softening=case["eps"], theta=case["theta"], dt=case["dt"],
                                substeps=case["substeps"], checkpoint_every=case["checkpoint"])
    return st


# ---- one pass -------------------------------------------------------------------------------


def run(st):
    case = st["case"]
    what = case["what"]
    if what in ("frame", "ensemble", "quasar"):
        sim = st["sim"]
        if what == "quasar":
            sim.step()
            k = sim.snapshot(0, max_bodies=st["rows"].shape[0], device_out=st["rows"].data_ptr())
            return {"count": k, "rows": st["rows"]}
        sim.substeps_async(case["substeps"])
        if st["out"] != "bodies":
            k = sim.snapshot(0 if st["out"] == "ue" else 1, device_out=st["rows"].data_ptr())
            return {"rows": st["rows"][:k]}
        rc = sim.lib.cosmosim_copy_bodies(sim.h, ptr(st["host"]), len(st["host"]))
        if rc:
            raise lib.CudaError(f"copy_bodies: {rc}")
        return _fields(st["host"], case.get("sph", False))
    if what == "step":
        lib.integrator_step(st["host"], case["dt"], 1.0, case["eps"], case["theta"], st["pool"],
                            int(case["sph"]))
        return {**_fields(st["host"], case["sph"]), "pool": _pool(st["pool"])}
    if what == "passes":
        b, pool = st["host"], st["pool"]
        _, cells = lib.octree_build(b, pool)
        lib.octree_compute_forces(pool, b, 1.0, case["eps"], case["theta"])
        lib.sph_compute_density(b, pool)
        lib.sph_compute_forces(b, pool)
        lib.sph_apply_cooling(b, case["dt"])
        return {**_fields(b, True), "cells": cells, "pool": _pool(pool)}
    if what == "diagnose":
        acc = st["sim"].direct_forces(st["idx"])
        return {"acc": acc, "energy": np.array(st["sim"].energy())}
    loss = st["adj"].forward(st["host"], st["target"])
    gx, gv = st["adj"].backward()
    return {"loss": np.array([loss]), "gx": gx, "gv": gv}


def _fields(b, sph):
    return {f: b[f] for f in STEP_FIELDS + (SPH_FIELDS if sph else ())}


def _pool(p):
    """The pool's columns (views of the caller's array)."""
    return {f: p[f] for f in NODE_DTYPE.names}


# ---- the same in 64 bits, by plain torch ------------------------------------------------------


class _Tree:
    """The octree of the reference (root cube of 1.01 times the extent, halved cells, one body a
    leaf), level by level. Per cell: size, parent, first child and their number, the body of a
    leaf; per level the cell of every body."""

    def __init__(self, x):
        n, dev = x.shape[0], x.device
        lo, hi = x.min(0).values, x.max(0).values
        hs = float((hi - lo).max()) * 0.5 * 1.01
        hs = hs if hs >= 1e-10 else 1.0
        centre = ((lo + hi) * 0.5).expand(n, 3).clone()
        who = torch.arange(n, device=dev)
        cell = torch.zeros(n, dtype=torch.long, device=dev)
        self.levels = [(who, cell)]
        size, leaf = [torch.full((1,), 2.0 * hs, dtype=torch.float64, device=dev)], []
        first, kids = [], []
        total = 1
        leaf.append(torch.full((1,), 0 if n == 1 else -1, dtype=torch.long, device=dev))
        key = torch.zeros((n, 3), dtype=torch.long, device=dev)  # octants, 21 levels a word
        base = 0
        if n == 1:
            first, kids = [torch.zeros(1, dtype=torch.long, device=dev)], [
                torch.zeros(1, dtype=torch.long, device=dev)]
        depth = 0
        while who.numel() and n > 1 and depth < 63:
            p = x[who]
            e, s, b = p[:, 0] >= centre[:, 0], p[:, 1] < centre[:, 1], p[:, 2] < centre[:, 2]
            q = e.long() + 2 * s.long() + 4 * b.long()
            step = torch.stack([torch.where(e, 0.5, -0.5), torch.where(s, -0.5, 0.5),
                                torch.where(b, -0.5, 0.5)], 1).double()
            centre = centre + step * hs
            key[who, depth // 21] |= q << (3 * (20 - depth % 21))
            hs *= 0.5
            u, inv, cnt = torch.unique((cell - base) * 8 + q, return_inverse=True,
                                       return_counts=True)
            par = u // 8  # in the level above
            above = size[-1].numel()
            k = torch.bincount(par, minlength=above)
            kids.append(k)
            first.append(total + torch.cumsum(k, 0) - k)
            size.append(torch.full((u.numel(),), 2.0 * hs, dtype=torch.float64, device=dev))
            lf = torch.full((u.numel(),), -1, dtype=torch.long, device=dev)
            single = cnt[inv] == 1
            lf[inv[single]] = who[single]
            leaf.append(lf)
            base, total = total, total + u.numel()
            cell = base + inv
            self.levels.append((who, cell))
            more = ~single
            who, cell, centre = who[more], cell[more], centre[more]
            depth += 1
        z = torch.zeros(total, dtype=torch.long, device=dev)
        self.first, self.kids = z.clone(), z.clone()
        f, k = torch.cat(first), torch.cat(kids)
        self.first[:f.numel()], self.kids[:k.numel()] = f, k
        self.s2 = torch.cat(size) ** 2
        self.leaf = torch.cat(leaf)
        self.total = total
        order = torch.arange(n, device=dev)
        for w in (2, 1, 0):
            order = order[torch.sort(key[order, w], stable=True).indices]
        self.order = order  # depth-first order of the bodies

    def moments(self, x, m):
        mass = torch.zeros(self.total, dtype=x.dtype, device=x.device)
        com = torch.zeros((self.total, 3), dtype=x.dtype, device=x.device)
        mx = m[:, None] * x
        for who, cell in self.levels:
            mass = mass.index_add(0, cell, m[who])
            com = com.index_add(0, cell, mx[who])
        return com / mass[:, None], mass

    def pairs(self, x, com, theta, lo, hi):
        """(body, cell) of every interaction of bodies lo..hi, in pieces."""
        i = torch.arange(lo, hi, device=x.device)
        c = torch.zeros_like(i)
        while i.numel():
            d2 = ((com[c] - x[i]) ** 2).sum(1)
            leaf = self.leaf[c]
            take = torch.where(leaf >= 0, leaf != i, (d2 > 0) & (self.s2[c] / d2 < theta * theta))
            yield i[take], c[take]
            down = ~take & (leaf < 0)
            i, c = i[down], c[down]
            k = self.kids[c]
            ends = torch.cumsum(k, 0)
            at = torch.arange(int(ends[-1]) if k.numel() else 0, device=x.device)
            i = torch.repeat_interleave(i, k)
            c = torch.repeat_interleave(self.first[c] - (ends - k), k) + at


def _gravity(x, m, eps, theta, G=1.0):
    t = _Tree(x)
    com, mass = t.moments(x, m)
    acc = torch.zeros_like(x)
    for lo in range(0, x.shape[0], 65536):
        for i, c in t.pairs(x, com, theta, lo, min(x.shape[0], lo + 65536)):
            d = com[c] - x[i]
            r2 = (d * d).sum(1) + eps * eps
            acc.index_add_(0, i, d * (G * mass[c] / (r2 * r2.sqrt()))[:, None])
    return acc, t


def _kernel(r, h):
    q = r / h
    norm = 8.0 / (math.pi * h ** 3)
    w = torch.where(q <= 0.5, norm * (1 - 6 * q * q + 6 * q ** 3), norm * 2 * (1 - q) ** 3)
    dw = torch.where(q <= 0.5, norm * (-12 * q + 18 * q * q) / h, norm * (-6 * (1 - q) ** 2) / h)
    none = (q > 1) | (h < 1e-10)
    return torch.where(none, 0.0, w), torch.where(none | (r < 1e-15), 0.0, dw)


def _neighbours(s, gas, order):
    """(gas body, neighbour) of the first 128 bodies within h in depth-first order."""
    xo = s["x"][order]
    for at in range(0, gas.numel(), 256):
        g = gas[at:at + 256]
        d2 = sum((xo[None, :, k] - s["x"][g][:, None, k]) ** 2 for k in range(3))
        near = d2 <= (s["h"][g] ** 2)[:, None]
        near &= torch.cumsum(near, 1, dtype=torch.int32) <= MAX_NB
        a, b = torch.nonzero(near, as_tuple=True)
        yield g[a], order[b]


def _density(s, order):
    gas = torch.nonzero((s["type"] == 1) & (s["m"] > 0)).flatten()
    rho, num = torch.zeros_like(s["m"]), torch.zeros_like(s["m"])
    for i, j in _neighbours(s, gas, order):
        r = (s["x"][i] - s["x"][j]).square().sum(1).sqrt()
        rho.index_add_(0, i, s["m"][j] * _kernel(r, s["h"][i])[0])
        num.index_add_(0, i, torch.ones_like(r))
    rho = rho.clamp(min=1e-15)
    h = s["h"].clone()
    grow, shrink = (num < 20) & (h < 50), (num > 48) & (h > 0.1)
    h = torch.where(grow, h * 1.2, torch.where(shrink, h * 0.8, h))
    s["h"][gas], s["rho"][gas] = h[gas], rho[gas]
    s["P"][gas] = (GAMMA - 1) * rho[gas] * s["u"][gas].clamp(min=1e-15)


def _pressure(s, order):
    gas = torch.nonzero((s["type"] == 1) & (s["m"] > 0)).flatten()
    cs = (GAMMA * s["P"] / (s["rho"] + 1e-15)).sqrt()
    pr = s["P"] / (s["rho"] ** 2 + 1e-15)
    acc = torch.zeros_like(s["x"])
    for i, j in _neighbours(s, gas, order):
        ok = (i != j) & (s["type"][j] == 1)
        i, j = i[ok], j[ok]
        d = s["x"][i] - s["x"][j]
        r = d.square().sum(1).sqrt()
        ok = r >= 1e-15
        i, j, d, r = i[ok], j[ok], d[ok], r[ok]
        h = 0.5 * (s["h"][i] + s["h"][j])
        vr = ((s["v"][i] - s["v"][j]) * d).sum(1)
        mu = h * vr / (r * r + 0.01 * h * h)
        visc = (-0.5 * (cs[i] + cs[j]) * mu + 2 * mu * mu) / (0.5 * (s["rho"][i] + s["rho"][j]) + 1e-15)
        visc = torch.where(vr < 0, visc, 0.0)
        f = s["m"][j] * (pr[i] + pr[j] + visc) * _kernel(r, h)[1] / r
        acc.index_add_(0, i, -f[:, None] * d)
    s["a"][gas] += 0.1 * acc[gas]


def _cool(s, dt):
    on = (s["type"] == 1) & (s["m"] > 0) & (s["u"] >= 1e-15) & (s["rho"] >= 1e-15)
    u = s["u"] / (1 + dt * COOL * s["rho"] * 0.5 / s["u"].clamp(min=1e-300).sqrt())
    u = u.clamp(min=GAS_MIN_U)
    s["u"] = torch.where(on, u, s["u"])
    s["P"] = torch.where(on, (GAMMA - 1) * s["rho"] * u, s["P"])


def _substep(s, case):
    s["v"] = s["v"] + 0.5 * s["a"] * case["dt"]
    s["x"] = s["x"] + s["v"] * case["dt"]
    s["a"], t = _gravity(s["x"], s["m"], case["eps"], case["theta"])
    if case.get("sph"):
        _density(s, t.order)
        _pressure(s, t.order)
    s["v"] = s["v"] + 0.5 * s["a"] * case["dt"]
    if case.get("sph"):
        _cool(s, case["dt"])


def _state(b, dev):
    col = lambda f: torch.tensor(np.ascontiguousarray(b[f]), device=dev).double()  # noqa: E731
    vec = lambda p: torch.stack([col(p + k) for k in "xyz"], 1)  # noqa: E731
    s = {"x": torch.stack([col(k) for k in "xyz"], 1), "v": vec("v"), "m": col("mass"),
         "type": col("type").long(), "u": col("internal_energy"), "h": col("smoothing_h"),
         "rho": col("density"), "P": col("pressure")}
    s["a"] = torch.zeros_like(s["x"])
    return s


def _state_fields(s, sph):
    out = {p + k: s[p or "x"][:, d] for p in ("", "v", "a") for d, k in enumerate("xyz")}
    if sph:
        out.update(density=s["rho"], pressure=s["P"], internal_energy=s["u"], smoothing_h=s["h"])
    return out


def _rows(s, out, b):
    cols = [s["x"], s["m"][:, None], s["v"], s["type"][:, None].double(), s["u"][:, None],
            s["rho"][:, None]]
    if out == "ue":
        more = [b[f] for f in ("lifetime", "luminosity", "spin_x", "spin_y", "spin_z")]
        more = torch.tensor(np.stack(more, 1), device=s["x"].device)
        cols += [more, torch.zeros_like(s["m"])[:, None]]
    return torch.cat(cols, 1)


def _adjoint(case, seed, dev):
    s = _state(_bodies(case, seed), dev)
    x0, v0, m = s["x"].requires_grad_(), s["v"].requires_grad_(), s["m"]
    target = torch.tensor(_target(case, seed), device=dev)

    def force(x):
        y = x.detach()
        t = _Tree(y)
        com, _ = t.moments(y, m)
        got = list(t.pairs(y, com, case["theta"], 0, y.shape[0]))
        i, c = (torch.cat([p[k] for p in got]) for k in (0, 1))  # the frozen lists
        com, mass = t.moments(x, m)
        d = com[c] - x[i]
        r2 = (d * d).sum(1) + case["eps"] ** 2
        return torch.zeros_like(x).index_add(0, i, d * (mass[c] / (r2 * r2.sqrt()))[:, None])

    step = lambda x, v, a: _leap(x, v, a, force, case["dt"])  # noqa: E731
    x, v = x0, v0
    a = torch.utils.checkpoint.checkpoint(force, x, use_reentrant=False)
    for _ in range(case["substeps"]):
        x, v, a = torch.utils.checkpoint.checkpoint(step, x, v, a, use_reentrant=False)
    loss = ((x - target) ** 2).sum(1).mean()
    gx, gv = torch.autograd.grad(loss, (x0, v0))
    return {"loss": loss.detach()[None], "gx": gx, "gv": gv}


def _leap(x, v, a, force, dt):
    v = v + 0.5 * a * dt
    x = x + v * dt
    a = force(x)
    return x, v + 0.5 * a * dt, a


def _diagnose(case, seed, dev):
    s = _state(_bodies(case, seed), dev)
    idx = torch.tensor(_sample(case, seed).astype(np.int64), device=dev)
    x, m, e2 = s["x"], s["m"], case["eps"] ** 2
    acc, pe = torch.zeros((idx.numel(), 3), dtype=torch.float64, device=dev), 0.0
    for at in range(0, idx.numel(), 256):
        d = x[None] - x[idx[at:at + 256]][:, None]
        r2 = d.square().sum(2) + e2
        acc[at:at + 256] = (d * (m / (r2 * r2.sqrt()))[:, :, None]).sum(1)
    n = x.shape[0]
    for at in range(0, n, 512):
        d2 = sum((x[None, :, k] - x[at:at + 512, k][:, None]) ** 2 for k in range(3))
        w = m[None] / (d2 + e2).sqrt()
        far = torch.arange(n, device=dev)[None] > torch.arange(at, min(n, at + 512), device=dev)[:, None]
        pe -= float((torch.where(far, w, 0.0).sum(1) * m[at:at + 512]).sum())
    ke = float((0.5 * m * s["v"].square().sum(1)).sum())
    return {"acc": acc, "energy": np.array([ke, pe])}


def exact(case, seed):
    what = case["what"]
    if what == "quasar":
        return None  # its random stream and index-ordered stages have no plain form
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if what == "adjoint":
        return _adjoint(case, seed, dev)
    if what == "diagnose":
        return _diagnose(case, seed, dev)
    b = _bodies(case, seed)
    if what == "ensemble":
        rows, at = [], 0
        for c in _counts(case):
            s = _state(b[at:at + c], dev)
            s["a"], _ = _gravity(s["x"], s["m"], case["eps"], case["theta"])
            for _ in range(case["substeps"]):
                _substep(s, case)
            rows.append(s)
            at += c
        s = {k: torch.cat([r[k] for r in rows]) for k in rows[0]}
        return {"rows": _rows(s, "render", b)} if case["prec"] == "fp32" else _state_fields(s, False)
    s = _state(b, dev)
    if what == "passes":
        s["a"], t = _gravity(s["x"], s["m"], case["eps"], case["theta"])
        _density(s, t.order)
        _pressure(s, t.order)
        _cool(s, case["dt"])
        return {**_state_fields(s, True), "cells": None, "pool": None}
    s["a"], _ = _gravity(s["x"], s["m"], case["eps"], case["theta"])
    for _ in range(case.get("substeps", 1)):
        _substep(s, case)
    if what == "step":
        return {**_state_fields(s, case["sph"]), "pool": None}
    return _state_fields(s, case["sph"]) if case["out"] == "bodies" else {
        "rows": _rows(s, case["out"], b)}
