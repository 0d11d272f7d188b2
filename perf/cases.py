"""Workloads that the framework's speed is judged by, with their 64-bit answers.

A case is one call pattern of a user's program, through the package's public
entry points:

* ``rk4``   RK4 steps through ``Context.rk4_step_host`` on a state that the
            program keeps in pinned host memory (its copies in and out are part
            of the pass), by the treecode or the direct sum, in mixed or double
            precision, with or without target clusters, with the fixed or the
            learned per-leaf parameters.
* ``rhs``   one right-hand side through ``Context.rhs`` on host arrays, as the
            reference's own time loop calls it, with or without the stream
            function.  Double precision.
* ``remesh`` device-resident RK4 steps, each followed by the regridding onto
            the icosahedral grid, then the state read back.
* ``ensemble`` uneven members advanced together, every member's state read back.

Particles are the vertices of the icosahedral grid, or (``grid`` 0) a jittered
spiral of any number of points, which no grid level and no tile divides.
Fields are Rossby-Haurwitz waves with Gaussian vortices drawn from the seed.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.abspath("fast-sphere-sum_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import fss_b200 as fss  # noqa: E402
from fss_b200 import selector  # noqa: E402

DT = 0.01  # days, the benchmark's step
OMEGA = 2 * math.pi
FLOPS_PER_PAIR = 23
VORTICES = 32


def _points(level):
    return 10 * 4 ** level + 2


def _rk4(name, n=0, level=None, fp64=False, tree=True, degree=8, theta=0.7, clusters=False, learned=False, steps=1):
    return {"name": name, "kind": "rk4", "grid": level is not None, "level": level or 0,
            "n": _points(level) if level is not None else n, "fp64": fp64, "tree": tree, "degree": degree,
            "theta": theta, "clusters": clusters, "learned": learned, "steps": steps}


def _rhs(name, n=0, level=None, tree=True, psi=False, degree=8, theta=0.7):
    return {"name": name, "kind": "rhs", "grid": level is not None, "level": level or 0,
            "n": _points(level) if level is not None else n, "fp64": True, "tree": tree, "degree": degree,
            "theta": theta, "clusters": False, "psi": psi}


def listed():
    return [
        # the smallest problem, called as the reference's loop calls it: launches and copies
        _rhs("rhs_direct_fp64_level3", level=3, tree=False),
        # a diagnostic right-hand side with the stream function, host arrays in and out
        _rhs("rhs_tree_psi_fp64_level6", level=6, psi=True),
        # small run of the default configuration (mixed treecode): a step is a chain of short launches
        _rk4("rk4_tree_mixed_level5", level=5, steps=2),
        # ragged particle count, default configuration
        _rk4("rk4_tree_mixed_100003", n=100003, steps=2),
        # the largest: the default configuration on the finest benchmark grid
        _rk4("rk4_tree_mixed_level8", level=8),
        # the benchmark's headline: learned per-leaf degree and acceptance, target clusters
        _rk4("rk4_learned_mixed_level8", level=8, clusters=True, learned=True),
        # double-precision treecode, n = 8, theta = 0.7, 163,842 particles
        _rk4("rk4_tree_fp64_level7", level=7, fp64=True),
        # the reference's cluster-cluster scheme at a higher degree
        _rk4("rk4_clusters_mixed_level7", level=7, degree=10, clusters=True, steps=2),
        # direct sums: the double-precision reference trajectory and the mixed one
        _rk4("rk4_direct_fp64_20011", n=20011, fp64=True, tree=False),
        _rk4("rk4_direct_mixed_level6", level=6, tree=False),
        # runs that put the particles back on the grid after every step
        {"name": "remesh_mixed_level7", "kind": "remesh", "level": 7, "n": _points(7), "degree": 8, "theta": 0.7,
         "steps": 2},
        # many uneven problems at once
        {"name": "ensemble_16_levels_4_to_7", "kind": "ensemble", "members": 16, "low": 4, "high": 7, "degree": 8,
         "theta": 0.7, "pick": 5, "steps": 1},
    ]


def _size(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["rk4"] * 7 + ["rhs"] * 2 + ["remesh", "ensemble"])
    degree, theta = rng.choice([6, 8, 8, 10]), rng.choice([0.6, 0.7, 0.7, 0.8])
    if kind == "ensemble":
        high = rng.randint(5, 7)
        case = {"kind": kind, "members": rng.randint(3, 20), "low": rng.randint(3, high), "high": high,
                "degree": degree, "theta": theta, "pick": rng.randint(0, 10 ** 6), "steps": rng.randint(1, 2)}
    elif kind == "remesh":
        level = rng.randint(4, 7)
        case = {"kind": kind, "level": level, "n": _points(level), "degree": degree, "theta": theta,
                "steps": rng.randint(1, 2)}
    elif kind == "rhs":
        tree = rng.random() < 0.7
        case = _rhs("", n=_size(rng, 642, 120000 if tree else 20000), tree=tree, psi=rng.random() < 0.5,
                    degree=degree, theta=theta)
    else:
        tree, fp64 = rng.random() < 0.75, rng.random() < 0.3
        if tree:
            level = rng.randint(4, 7 if fp64 else 8)
            n = _size(rng, 2000, 160000 if fp64 else 655362)
            learned = not fp64 and level >= 7 and rng.random() < 0.4
            case = _rk4("", n=n, level=level if learned or rng.random() < 0.4 else None, fp64=fp64, degree=degree,
                        theta=theta, clusters=learned or rng.random() < 0.4, learned=learned)
        else:
            case = _rk4("", n=_size(rng, 700, 20000 if fp64 else 60000), fp64=fp64, tree=False)
        case["steps"] = 2 if case["n"] <= 200000 and rng.random() < 0.5 else 1
    case.pop("name", None)
    return case


# ------------------------------------------------------------------- inputs

@functools.lru_cache(maxsize=None)
def _grid(level):
    """Vertices, faces and areas of a level: files that a user's program reads once."""
    xyz, faces = fss.icos_grid(level)
    s = np.zeros((xyz.shape[0], 5))
    s[:, :3] = xyz
    return xyz, faces, fss.area_init(s, faces)


def _spiral(n, rng):
    """n points spread evenly over the sphere, moved by up to a third of their spacing."""
    i = np.arange(n) + 0.5
    z = 1 - 2 * i / n
    lon = math.pi * (1 + 5 ** 0.5) * i
    r = np.sqrt(1 - z * z)
    x = np.stack([r * np.cos(lon), r * np.sin(lon), z], 1)
    x += rng.uniform(-1, 1, x.shape) * (math.sqrt(4 * math.pi / n) / 3 / math.sqrt(3))
    x /= np.linalg.norm(x, axis=1, keepdims=True)
    return x[rng.permutation(n)], np.full(n, 4 * math.pi / n)


def _field(xyz, area, rng, vortices):
    """Rossby-Haurwitz wave plus Gaussian vortices, mean vorticity removed; tracer 2 + latitude."""
    s = np.empty((xyz.shape[0], 5))
    s[:, :3] = xyz
    lat, lon = np.arcsin(np.clip(xyz[:, 2], -1, 1)), np.arctan2(xyz[:, 1], xyz[:, 0])
    w = fss.RH_AMP * rng.uniform(0.9, 1.1)
    zeta = 2 * w * xyz[:, 2] - 30 * w * np.cos(lat) ** 4 * xyz[:, 2] * np.cos(4 * lon)
    for _ in range(vortices):
        c = rng.standard_normal(3)
        c /= np.linalg.norm(c)
        near = np.flatnonzero(xyz @ c > math.cos(0.65))
        zeta[near] += (math.pi * 2 ** 0.5 * rng.standard_normal()
                       * np.exp(-(np.arccos(np.clip(xyz[near] @ c, -1, 1)) / 0.1) ** 2))
    s[:, 3] = zeta - np.sum(zeta * area) / np.sum(area)
    s[:, 4] = 2 + lat
    return s


def _inputs(case, seed):
    """[(state (N, 5), area (N,))] of the case's problem, or of its members."""
    if case["kind"] == "ensemble":
        levels = np.random.default_rng(case["pick"]).integers(case["low"], case["high"] + 1, case["members"])
        return [_one(_points(int(k)), int(k), np.random.default_rng([seed, m]), 8) for m, k in enumerate(levels)]
    on_grid = case["kind"] == "remesh" or case["grid"]
    return [_one(case["n"], case["level"] if on_grid else None, np.random.default_rng(seed), VORTICES)]


def _one(n, level, rng, vortices):
    if level is None:
        xyz, area = _spiral(n, rng)
    else:
        xyz, _, area = _grid(level)
    return _field(xyz, area, rng, vortices), area


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.copy_(torch.from_numpy(a))
    return t


# -------------------------------------------------------------------- passes

def prepare(case, seed):
    parts = _inputs(case, seed)
    if case["kind"] == "ensemble":
        ens = fss.Ensemble(degree=case["degree"], theta=case["theta"])
        for s, a in parts:
            ens.add(s, a)
        ens.build()
        return {"case": case, "ens": ens}
    s, a = parts[0]
    options = {"degree": case["degree"], "theta": case["theta"]}
    if case["kind"] == "remesh":
        ctx = fss.Context(precision=fss.PREC_MIXED, **options)
    else:
        options["cluster_targets"] = int(case["clusters"])
        if case.get("learned"):
            options["list_mode"] = fss.LIST_LEAF
        ctx = fss.Context(method=fss.METHOD_TREECODE if case["tree"] else fss.METHOD_DIRECT,
                          precision=fss.PREC_FP64 if case["fp64"] else fss.PREC_MIXED, **options)
    ctx.set_particles(s, a)
    if case.get("learned"):
        selector.apply(ctx, tol=1e-6, safety=2.0)
    state = {"case": case, "ctx": ctx, "area": a}
    if case["kind"] == "remesh":
        state["tris"] = _grid(case["level"])[1]
    elif case["kind"] == "rk4":
        state["pinned"] = _pinned(s)
        state["state"] = state["pinned"].numpy()
    else:
        state["state"] = s
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "ensemble":
        ens = state["ens"]
        ens.rk4_step(DT, nsteps=case["steps"])
        return [ens.get_state(m) for m in range(case["members"])]
    ctx = state["ctx"]
    if case["kind"] == "rhs":
        return ctx.rhs(state["state"], state["area"], psi=case["psi"])
    if case["kind"] == "remesh":
        for _ in range(case["steps"]):
            ctx.rk4_step(DT)
            ctx.remesh_current(state["tris"])
        return ctx.get_state()
    return ctx.rk4_step_host(state["state"], DT, nsteps=case["steps"])


# ---------------------------------------------------------------------- work

@functools.lru_cache(maxsize=None)
def _pairs(n, level, tree, degree, theta, clusters, learned):
    """Interactions of one right-hand side: all pairs of the direct sum, or
    those that the treecode's traversal accepts."""
    if not tree:
        return float(n) * (n - 1)
    case = {"kind": "rk4", "grid": level is not None, "level": level, "n": n, "fp64": False, "tree": True,
            "degree": degree, "theta": theta, "clusters": clusters, "learned": learned}
    info = prepare(case, 1)["ctx"].tree_info()
    return sum(info[k + "_interactions"] for k in ("pp", "pc", "cp", "cc"))


def work(case):
    """Pair interactions of the method that the case asks for (a treecode's
    traversal fixes them), and each particle's state and area read and its
    state written once per right-hand side."""
    if case["kind"] == "ensemble":
        pairs = n = 0
        for k in np.random.default_rng(case["pick"]).integers(case["low"], case["high"] + 1, case["members"]):
            n += _points(int(k))
            pairs += _pairs(_points(int(k)), int(k), True, case["degree"], case["theta"], False, False)
    else:
        n = case["n"]
        on_grid = case["kind"] == "remesh" or case["grid"]
        pairs = _pairs(n, case["level"] if on_grid else None, case.get("tree", True), case["degree"], case["theta"],
                       case.get("clusters", False), case.get("learned", False))
    evaluations = 1 if case["kind"] == "rhs" else 4 * case["steps"]
    return {"bytes": evaluations * n * 8 * 11.0, "flops": evaluations * pairs * FLOPS_PER_PAIR}


# -------------------------------------------------------------- 64-bit answers

def _sums(x, w, psi=False, block=8192):
    """Direct sums over all pairs j != i: u (N, 3) and, when asked, psi (N,).
    1 / (1 - x.y) is symmetric, so each block of pairs serves both sides."""
    n = x.shape[0]
    one = torch.ones(n, 1, dtype=x.dtype, device=x.device)
    left, right = torch.cat([x, one], 1), torch.cat([-x, one], 1)
    charge = w[:, None] * x
    acc, logs = torch.zeros_like(x), torch.zeros_like(w)
    for i in range(0, n, block):
        a = slice(i, min(i + block, n))
        for j in range(i, n, block):
            b = slice(j, min(j + block, n))
            if n <= 50000:  # differences of the coordinates, no cancellation
                g = sum((x[a, k, None] - x[None, b, k]) ** 2 for k in range(3)).mul_(0.5)
            else:           # neighbours are still 1e-5 apart: 1 - x.y to 1e-11
                g = left[a] @ right[b].T
            if i == j:
                g.fill_diagonal_(math.inf)
            if psi:
                lg = g.log()
                if i == j:
                    lg.fill_diagonal_(0.0)
                logs[a] += lg @ w[b]
                if i != j:
                    logs[b] += lg.T @ w[a]
            g.reciprocal_()
            acc[a] += g @ charge[b]
            if i != j:
                acc[b] += g.T @ charge[a]
    u = torch.linalg.cross(x, acc).mul_(-1 / (4 * math.pi))
    return (u, logs.mul_(-1 / (4 * math.pi))) if psi else u


def _rate(s, area):
    k = torch.zeros_like(s)
    k[:, :3] = _sums(s[:, :3].contiguous(), s[:, 3] * area)
    k[:, 3] = -2 * OMEGA * k[:, 2]
    return k


def _onto_sphere(s):
    s = s.clone()
    z = s[:, 2].clone()
    s[:, :3] /= torch.linalg.vector_norm(s[:, :3], dim=1, keepdim=True)
    s[:, 3] -= 2 * OMEGA * (s[:, 2] - z)
    return s


def _steps(s, area, count):
    for _ in range(count):
        k1 = _rate(s, area)
        k2 = _rate(_onto_sphere(s + DT / 2 * k1), area)
        k3 = _rate(_onto_sphere(s + DT / 2 * k2), area)
        k4 = _rate(_onto_sphere(s + DT * k3), area)
        s = _onto_sphere(s + DT / 6 * (k1 + 2 * k2 + 2 * k3 + k4))
    return s


def exact(case, seed):
    if case["kind"] == "remesh":
        return None
    out = []
    for s, a in _inputs(case, seed):
        s, a = (torch.from_numpy(v).to("cuda") for v in (s, a))
        if case["kind"] != "rhs":
            out.append(_steps(s, a, case["steps"]).cpu().numpy())
        elif case["psi"]:
            u, p = _sums(s[:, :3].contiguous(), s[:, 3] * a, psi=True)
            k = torch.zeros_like(s)
            k[:, :3], k[:, 3] = u, -2 * OMEGA * u[:, 2]
            return k.cpu().numpy(), p.cpu().numpy()
        else:
            return _rate(s, a).cpu().numpy()
    return out if case["kind"] == "ensemble" else out[0]
