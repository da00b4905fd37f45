"""The work that users of this package have it do, as cases that can be timed.

``listed()`` gives the cases, ``draw(rng)`` one more of the same ranges, ``prepare`` the
inputs that a program holds before the call, ``run`` one pass through the public entry
points, ``work`` the bytes and operations that the pass cannot do without and ``exact``
the same results from plain torch in 64 bits.

Units: kpc, km/s, Msun, Myr.  Systems are the package's own seeded ones: Plummer spheres
(b = 1 pc, 1e6 Msun, eps = 0.05 pc, dt = 0.005 Myr) for the direct sum, ensembles and
gradients, and the Hernquist spheroid plus exponential disk (eps = 0.1 kpc, dt = 0.5 Myr)
for the tree.  Masses are equal (as every generator makes them) or, with "masses":
"mixed", spread over about a factor of ten (two components of different resolution).
"""
import math

import numpy as np
import torch

import gravhopper_gb300 as gh
from gravhopper_gb300 import engine, ics
from gravhopper_gb300.adjoint import rollout
from gravhopper_gb300.ensemble import Ensemble

ACCEL = 4.398600412921223e-09  # G Msun / kpc^2 in km/s/Myr
KMS_MYR = 1.022712165045695e-03  # (km/s) Myr in kpc


def listed():
    return [
        # a short script's force call, NumPy arrays in and out (the drop-in for the reference's
        # C extension): copies, launches and latency are most of it
        {"name": "host_direct_n500", "kind": "host", "algorithm": "direct", "n": 500, "theta": 0.7},
        # the reference's own example size through Simulation, every snapshot kept: direct sum
        {"name": "sim_direct_n2000", "kind": "sim", "algorithm": "direct", "precision": "fp64", "n": 2000,
         "theta": 0.7, "steps": 20},
        # the same through Simulation's defaults: Barnes-Hut tree, 64 bits
        {"name": "sim_tree_n2000", "kind": "sim", "algorithm": "tree", "precision": "fp64", "n": 2000,
         "theta": 0.7, "steps": 10},
        # one tree force of a medium galaxy model, an odd size
        {"name": "tree_fp64_n60013", "kind": "tree", "precision": "fp64", "n": 60013, "points": 0, "theta": 0.7,
         "system": "disk"},
        # field at arbitrary points (a rotation curve, a map, test particles) of a larger model
        {"name": "tree_points_fp64_n250000", "kind": "tree", "precision": "fp64", "n": 250000, "points": 30011,
         "theta": 0.5, "system": "disk"},
        # a leapfrog step of the million-particle galaxy in 64 bits
        {"name": "tree_step_fp64_n1048576", "kind": "tree_step", "precision": "fp64", "n": 1048576, "theta": 0.7,
         "steps": 1},
        # the same in the mixed form
        {"name": "tree_step_mixed_n1048576", "kind": "tree_step", "precision": "mixed", "n": 1048576, "theta": 0.5,
         "steps": 1},
        # the direct sum in 64 bits: one force, two components of different particle mass
        {"name": "direct_fp64_n65536", "kind": "direct", "precision": "fp64", "n": 65536, "points": 0,
         "masses": "mixed"},
        # a leapfrog step of the mixed direct sum (drawn cases: its forces, at particles and points)
        {"name": "step_mixed_n262144", "kind": "step", "precision": "mixed", "n": 262144, "steps": 1},
        # 512 spheres of 256 to 8192 particles in one ensemble
        {"name": "ensemble_512", "kind": "ensemble", "systems": 512, "nmin": 256, "nmax": 8192, "steps": 4},
        # gradients of a rollout's loss with respect to its initial conditions and masses
        {"name": "rollout_mixed_n16384", "kind": "rollout", "precision": "mixed", "n": 16384, "steps": 10, "every": 5},
        # the potential behind every energy check of a run
        {"name": "potential_n65536", "kind": "potential", "n": 65536, "masses": "equal"},
    ]


def draw(rng):
    def log_int(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["host", "sim", "sim", "tree", "tree", "tree_step", "direct", "step", "ensemble", "rollout",
                       "potential"])
    c = {"kind": kind}
    if kind in ("host", "sim"):
        c["algorithm"] = rng.choice(["direct", "tree"])
        c["theta"] = rng.choice([0.5, 0.7, 1.0])
        c["n"] = log_int(64, 8192)
        if kind == "sim":
            c["precision"] = rng.choice(["fp64", "fp64", "mixed"])
            c["steps"] = rng.randint(5, 20)
    elif kind in ("tree", "tree_step"):
        c["precision"] = rng.choice(["fp64", "fp64", "mixed"])
        c["theta"] = rng.choice([0.5, 0.7, 1.0])
        c["n"] = log_int(8192, 600000)
        if kind == "tree":
            c["points"] = rng.choice([0, log_int(100, 100000)])
            c["system"] = rng.choice(["disk", "plummer"])
        else:
            c["steps"] = rng.randint(1, 3)
    elif kind == "direct":
        c["precision"] = rng.choice(["fp64", "mixed"])
        c["n"] = log_int(1000, 65536 if c["precision"] == "fp64" else 200000)
        c["points"] = rng.choice([0, log_int(10, 50000)])
        c["masses"] = rng.choice(["equal", "mixed"])
    elif kind == "step":
        c["precision"] = rng.choice(["fp64", "mixed"])
        c["n"] = log_int(4096, 50000 if c["precision"] == "fp64" else 300000)
        c["steps"] = 1 if c["n"] > 20000 else rng.randint(1, 5)
    elif kind == "ensemble":
        c["systems"] = log_int(16, 400)
        c["nmin"], c["nmax"] = log_int(64, 1024), log_int(2048, 8192)
        c["steps"] = rng.randint(1, 6)
    elif kind == "rollout":
        c["precision"] = rng.choice(["fp64", "mixed"])
        c["n"] = log_int(256, 4096 if c["precision"] == "fp64" else 16384)
        c["steps"] = rng.randint(3, 10)
        c["every"] = rng.randint(2, 5)
    else:
        c["n"] = log_int(1000, 65536)
        c["masses"] = rng.choice(["equal", "mixed"])
    return c


# ---- inputs --------------------------------------------------------------------------
def _system(case, seed):
    """Initial conditions on the host, the softening and the step."""
    n = case["n"]
    if case["kind"] in ("host", "sim", "direct", "step", "rollout", "potential") or case.get("system") == "plummer":
        ic, eps, dt = ics.plummer(n, seed=seed), 5e-5, 0.005
    else:
        ic, eps, dt = ics.hernquist_disk(n, seed=seed), 0.1, 0.5
    if case.get("masses") == "mixed":
        w = np.exp(np.random.default_rng(seed + 1).uniform(0.0, math.log(10.0), n))
        ic["mass"] = w * (ic["mass"].sum() / w.sum())
    return ic, eps, dt


def _points(case, ic, seed):
    """Field points: around particles (90 %) and on rays out of the system."""
    k = case["points"]
    rng = np.random.default_rng(seed + 2)
    p = ic["pos"][rng.integers(0, len(ic["pos"]), k)] * rng.uniform(0.8, 1.2, (k, 1))
    far = rng.random(k) < 0.1
    p[far] *= rng.uniform(1.0, 10.0, (int(far.sum()), 1))
    return p


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda")


def _sizes(case):
    """Particles of each system of an ensemble: log-uniform, the same for every seed."""
    rng = np.random.default_rng(case["systems"])
    ns = np.exp(rng.uniform(np.log(case["nmin"]), np.log(case["nmax"] + 1), size=case["systems"])).astype(np.int64)
    return np.clip(ns, case["nmin"], case["nmax"])


def _spheres(case, seed):
    """The systems of an ensemble: b from 0.5 to 2 pc, eps and dt scaled with it."""
    rng = np.random.default_rng(seed)
    out = []
    for n in _sizes(case):
        b = rng.uniform(0.5e-3, 2.0e-3)
        out.append(dict(ics.plummer(int(n), b=b, seed=int(rng.integers(1 << 62))), eps=0.05 * b, dt=0.005 * (b / 1e-3) ** 1.5))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "ensemble":
        s["ens"] = Ensemble(_spheres(case, seed))
        s["pos"], s["vel"] = s["ens"].pos.clone(), s["ens"].vel.clone()
        return s
    ic, s["eps"], s["dt"] = _system(case, seed)
    if kind in ("host", "sim"):
        s["ic"] = ic
        return s
    s["pos"], s["vel"], s["mass"] = (_device(ic[k]) for k in ("pos", "vel", "mass"))
    if case.get("points"):
        s["points"] = _device(_points(case, ic, seed))
    if kind == "rollout":
        noise = np.random.default_rng(seed + 3).normal(0.0, 1e-3, ic["pos"].shape)
        s["target"] = _device(ic["pos"] * (1.0 + noise))
    return s


# ---- one pass ------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "host":
        snap = {"pos": s["ic"]["pos"], "mass": s["ic"]["mass"]}
        if case["algorithm"] == "direct":
            return gh.grav.direct_summation(snap, s["eps"])
        return gh.grav.tree_force(snap, s["eps"], theta=case["theta"])
    if kind == "sim":
        sim = gh.Simulation(dt=s["dt"], eps=s["eps"], algorithm=case["algorithm"], theta=case["theta"],
                            precision=case["precision"])
        sim.add_IC(s["ic"])
        sim.run(case["steps"])
        return {"positions": sim.positions, "velocities": sim.velocities}
    if kind == "tree":
        return engine.tree_force(s["pos"], s["mass"], s["eps"], case["theta"], force_pos=s.get("points"),
                                 precision=case["precision"])
    if kind == "direct":
        return engine.direct_force(s["pos"], s["mass"], s["eps"], force_pos=s.get("points"),
                                   precision=case["precision"])
    if kind in ("tree_step", "step"):
        x, v = s["pos"].clone(), s["vel"].clone()
        engine.run_dkd(x, v, s["mass"], case["steps"], s["dt"], s["eps"],
                       algorithm="tree" if kind == "tree_step" else "direct", precision=case["precision"],
                       theta=case.get("theta", 0.7))
        return {"pos": x, "vel": v}
    if kind == "ensemble":
        e = s["ens"]
        e.pos.copy_(s["pos"])
        e.vel.copy_(s["vel"])
        e.run(case["steps"])
        return {"pos": e.pos, "vel": e.vel}
    if kind == "rollout":
        x0, v0, m = (s[k].detach().requires_grad_() for k in ("pos", "vel", "mass"))
        x, v = rollout(x0, v0, m, case["steps"], s["dt"], s["eps"], checkpoint_every=case["every"],
                       precision=case["precision"])
        loss = ((x - s["target"]) ** 2).mean()
        loss.backward()
        return {"pos": x.detach(), "vel": v.detach(), "grad_pos": x0.grad, "grad_vel": v0.grad, "grad_mass": m.grad}
    return engine.potential(s["pos"], s["mass"], s["eps"])


# ---- what a pass cannot do without ------------------------------------------------------
def work(case):
    """Bytes: state or inputs read once, results written once.  Operations: 20 per pair
    interaction of a force (the usual count), 12 of a potential, 60 of a force's gradient;
    a tree's interactions per particle are about 1350 (0.7 / theta)^2.7 log2(n) / 20,
    counted on the galaxy model at a million particles."""
    kind = case["kind"]
    if kind == "ensemble":
        ns = _sizes(case).astype(np.float64)
        return {"bytes": 104.0 * float(ns.sum()), "flops": 20.0 * case["steps"] * float((ns * ns).sum())}
    n = float(case["n"])
    targets = float(case.get("points") or n)
    if kind in ("tree", "tree_step") or case.get("algorithm") == "tree":
        each = min(n, 1350.0 * (0.7 / case["theta"]) ** 2.7 * math.log2(n) / 20.0)
    else:
        each = n
    steps = case.get("steps", 1)
    flops = 20.0 * targets * each * steps
    if kind in ("host", "tree", "direct"):
        return {"bytes": 32.0 * n + 24.0 * targets + (24.0 * targets if case.get("points") else 0.0), "flops": flops}
    if kind == "potential":
        return {"bytes": 40.0 * n, "flops": 12.0 * n * n}
    if kind == "sim":
        return {"bytes": 56.0 * n + 48.0 * n * steps, "flops": flops}
    if kind == "rollout":
        return {"bytes": 56.0 * n + 104.0 * n, "flops": steps * (20.0 + 60.0) * n * n}
    return {"bytes": 104.0 * n, "flops": flops}


# ---- the same results in plain 64-bit torch ------------------------------------------------
PAIRS = 2e11  # direct sums of more pairs than this take too long here
BLOCK = 3e7   # pairs held at once


def _blocks(nt, n):
    k = max(1, int(BLOCK // max(n, 1)))
    for a in range(0, nt, k):
        yield a, min(nt, a + k)


def _inv_cube(s):
    r = torch.where(s > 0, s, torch.ones_like(s)).rsqrt()
    return torch.where(s > 0, r * r * r, torch.zeros_like(s))


def _direct(x, m, eps, t=None):
    t = x if t is None else t
    out = torch.empty_like(t)
    for a, b in _blocks(len(t), len(x)):
        d = [x[None, :, k] - t[a:b, None, k] for k in range(3)]
        w = _inv_cube(d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps * eps) * m
        for k in range(3):
            out[a:b, k] = (w * d[k]).sum(1)
    return out


def _potential(x, m, eps):
    out = torch.empty_like(m)
    for a, b in _blocks(len(x), len(x)):
        s = sum((x[None, :, k] - x[a:b, None, k]) ** 2 for k in range(3)) + eps * eps
        w = m * s.rsqrt()
        w[torch.arange(b - a, device=x.device), torch.arange(a, b, device=x.device)] = 0.0
        out[a:b] = -w.sum(1)
    return out


def _vjp(x, m, eps, lam):
    """(lam . da/dx, lam . da/dm) of the direct sum."""
    gx, gm = torch.empty_like(x), torch.empty_like(m)
    for a, b in _blocks(len(x), len(x)):
        d = [x[None, :, k] - x[a:b, None, k] for k in range(3)]
        s = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps * eps
        q = s.rsqrt() ** 3
        u = [m[a:b, None] * lam[None, :, k] - m[None, :] * lam[a:b, None, k] for k in range(3)]
        p = 3.0 * q / s * (d[0] * u[0] + d[1] * u[1] + d[2] * u[2])
        for k in range(3):
            gx[a:b, k] = (q * u[k] - p * d[k]).sum(1)
        gm[a:b] = -(q * (d[0] * lam[None, :, 0] + d[1] * lam[None, :, 1] + d[2] * lam[None, :, 2])).sum(1)
    return gx, gm


def _tree(x, m, eps, theta, t=None):
    """Barnes-Hut with one particle per leaf: root cube from the extents (+ eps), cells
    halved in the order x > c, a cell accepted where size / distance to its centre < theta."""
    dev, n = x.device, len(x)
    lo, hi = x.min(0).values.tolist(), x.max(0).values.tolist()
    size = (hi[0] - lo[0]) + eps
    for k in (1, 2):
        if hi[k] - lo[k] > size:
            size = (hi[k] - lo[k]) + eps
    # levels[L]: (centres, size, com, mass, children: start, count) of the cells of two or more
    cen = torch.tensor([[0.5 * (lo[k] + hi[k]) for k in range(3)]], dtype=x.dtype, device=dev)
    ids, cell, levels = torch.arange(n, device=dev), torch.zeros(n, dtype=torch.int64, device=dev), []
    while len(ids):
        nc = len(cen)
        mass = torch.zeros(nc, dtype=x.dtype, device=dev).index_add_(0, cell, m[ids])
        mom = torch.zeros(nc, 3, dtype=x.dtype, device=dev).index_add_(0, cell, m[ids, None] * x[ids])
        right = x[ids] > cen[cell]
        key = cell * 8 + right[:, 0].long() + 2 * right[:, 1].long() + 4 * right[:, 2].long()
        kids, inv, cnt = torch.unique(key, return_inverse=True, return_counts=True)
        single = cnt == 1
        inner = torch.cumsum((~single).long(), 0) - 1  # row of the kid among the next level's cells
        link = inner.clone()
        lone = single[inv]
        link[inv[lone]] = -1 - ids[lone]  # a leaf: its particle
        number = torch.bincount(kids // 8, minlength=nc)
        levels.append((cen, size, mom / mass[:, None], mass, torch.cumsum(number, 0) - number, number, link))
        off = 0.25 * size
        up = torch.stack([(kids >> k) & 1 for k in range(3)], 1).bool()
        nxt = torch.where(up, cen[kids // 8] + off, cen[kids // 8] - off)
        cen, size = nxt[~single], 0.5 * size
        cell, ids = inner[inv[~lone]], ids[~lone]
    targets = x if t is None else t
    out = torch.zeros_like(targets)

    def add(who, pos, mass):
        d = pos - targets[who]
        f = _inv_cube(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2] + eps * eps) * mass
        out.index_add_(0, who, f[:, None] * d)

    for a in range(0, len(targets), 60000):
        who = torch.arange(a, min(a + 60000, len(targets)), device=dev)
        at = torch.zeros_like(who)
        for cen, size, com, mass, start, number, link in levels:
            d = cen[at] - targets[who]
            near = size / torch.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]) < theta
            add(who[near], com[at[near]], mass[at[near]])
            who, at = who[~near], at[~near]
            k = number[at]
            row = torch.repeat_interleave(start[at] - (torch.cumsum(k, 0) - k), k) + torch.arange(int(k.sum()), device=dev)
            who, kid = torch.repeat_interleave(who, k), link[row]
            leaf = kid < 0
            add(who[leaf], x[-1 - kid[leaf]], m[-1 - kid[leaf]])
            who, at = who[~leaf], kid[~leaf]
            if not len(who):
                break
    return out


def _leapfrog(x, v, steps, dt, force):
    for _ in range(steps):
        xh = x + 0.5 * dt * KMS_MYR * v
        v = v + dt * ACCEL * force(xh)
        x = xh + 0.5 * dt * KMS_MYR * v
        yield xh, x, v


def exact(case, seed):
    kind = case["kind"]
    n = case.get("n", 0)
    if kind == "ensemble":
        xs, vs = [], []
        for s in _spheres(case, seed):
            x, v, m = (_device(s[k]) for k in ("pos", "vel", "mass"))
            for _, x, v in _leapfrog(x, v, case["steps"], s["dt"], lambda p: _direct(p, m, s["eps"])):
                pass
            xs.append(x)
            vs.append(v)
        return {"pos": torch.cat(xs), "vel": torch.cat(vs)}
    if kind in ("direct", "step") and float(n) * float(case.get("points") or n) * case.get("steps", 1) > PAIRS:
        return None
    ic, eps, dt = _system(case, seed)
    x, v, m = (_device(ic[k]) for k in ("pos", "vel", "mass"))
    t = _device(_points(case, ic, seed)) if case.get("points") else None
    tree = kind in ("tree", "tree_step") or case.get("algorithm") == "tree"

    def force(p, at=None):
        return _tree(p, m, eps, case["theta"], at) if tree else _direct(p, m, eps, at)

    if kind == "host":
        return ACCEL * force(x).cpu().numpy()
    if kind in ("tree", "direct"):
        return force(x, t)
    if kind == "potential":
        return _potential(x, m, eps)
    x0, v0 = x, v
    trail = list(_leapfrog(x, v, case["steps"], dt, force))
    if kind == "sim":
        return {"positions": torch.stack([x0] + [q[1] for q in trail]).cpu().numpy(),
                "velocities": torch.stack([v0] + [q[2] for q in trail]).cpu().numpy()}
    _, x, v = trail[-1]
    if kind != "rollout":
        return {"pos": x, "vel": v}
    noise = np.random.default_rng(seed + 3).normal(0.0, 1e-3, ic["pos"].shape)
    xb = 2.0 * (x - _device(ic["pos"] * (1.0 + noise))) / x.numel()
    vb, mb, c = torch.zeros_like(v), torch.zeros_like(m), 0.5 * dt * KMS_MYR
    for xh, _, _ in reversed(trail):
        w = vb + c * xb
        gx, gm = _vjp(xh, m, eps, dt * ACCEL * w)
        xb, mb = xb + gx, mb + gm
        vb = w + c * xb
    return {"pos": x, "vel": v, "grad_pos": xb, "grad_vel": vb, "grad_mass": mb}
