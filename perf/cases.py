"""The work that a user of this framework has it do, as cases to time.

A case is a dict of plain values; `prepare` makes what a program holds before
the call (points, meshes, displacements, output tables, all from the seed),
`run` is one pass through the public classes, `work` the bytes and operations
of a pass that no implementation can do without, `exact` the computed numbers
of the first pass in 64 bits.

Coordinates lie in the unit square scaled by 2^13 (the scale of the package's
own workloads).  Uniform points are drawn with one point per unit cell, so that
the Morton order the build sorts them into is unique; the precision-stress set
is the package's own.
"""
import math

import numpy as np
import torch

import mcleap_gb300 as M
from mcleap_gb300 import workloads
from mcleap_gb300.batch import build_mesh

L = 8192.0
HI = np.nextafter(np.float32(L), np.float32(0))
RING = 32      # slots of a ring row: a count and up to 31 neighbours
NEAR = 32      # slots of a neighbour row at r = 2 x spacing (12.6 on average)
FAR = 64       # ... at r = 3 x spacing (28.3 on average)


def listed():
    return [
        # A small mesh stepped interactively: walk, settle, untangle, Delaunay
        # and rings, the counters of every step read back.
        {"name": "walk-1k", "kind": "walk", "n": 1000, "sigma": 0.1, "stats": True, "near": False},
        # The plain method's small configuration: 10,000 points, a random walk
        # of 0.1 x spacing that tangles the mesh, then the neighbours within 2 x
        # spacing of every point from the uniform grid.
        {"name": "plain-10k", "kind": "walk", "n": 10000, "sigma": 0.1, "stats": True, "near": True},
        # One mesh of the repair benchmark's size: 137 thousand faces turned
        # over by every step.
        {"name": "walk-1m", "kind": "walk", "n": 1000000, "sigma": 0.1, "stats": False, "near": False},
        # The headline configuration: a million points advected by the
        # Taylor-Green vortex, 0.5 x spacing at most, and the one-rings.
        {"name": "advect-1m", "kind": "advect", "n": 1000000, "frac": 0.5},
        # An advected mesh of a test's size, odd.
        {"name": "advect-20k", "kind": "advect", "n": 20011, "frac": 0.5},
        # The precision-stress set: a jittered lattice (cocircular quads),
        # clusters and uniform points, walking 0.05 x spacing.
        {"name": "stress-500k", "kind": "stress", "n": 500000, "sigma": 0.05},
        # A batch of independent meshes of uneven size, walk to neighbours.
        {"name": "batch-96", "kind": "batch", "meshes": 96, "lo": 100, "hi": 100000, "sigma": 0.1},
        # One iteration of the server: half of the resident meshes step (an
        # aggregation with few walkers left), query lists on the others.
        {"name": "serve-48", "kind": "serve", "meshes": 48, "lo": 1000, "hi": 200000, "walkers": 0.02, "queries": 60000},
        # Fixed-radius neighbours of a million points on the torus, r = 3 x
        # spacing, in the points' own order: the headline's query.
        {"name": "frnn-torus-1m", "kind": "frnn", "n": 1000000, "r": 3.0, "periodic": True, "inplace": False},
        # Rings and nearest ring neighbours of a static mesh, row layout.
        {"name": "rings-500k", "kind": "rings", "n": 500009, "row": True},
        # The initial triangulation of a mesh that is admitted: host points to
        # rings.
        {"name": "build-100k", "kind": "build", "n": 100000},
        # The periodic mesh: advection with a drift, points wrap every step.
        {"name": "torus-200k", "kind": "torus", "n": 200000, "frac": 0.5},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["walk", "walk", "advect", "stress", "batch", "serve", "frnn", "rings", "build", "torus"])
    if kind == "walk":
        return {"kind": kind, "n": _log_uniform(rng, 300, 900000), "sigma": round(rng.uniform(0.02, 0.15), 3),
                "stats": rng.random() < 0.5, "near": rng.random() < 0.5}
    if kind == "advect":
        return {"kind": kind, "n": _log_uniform(rng, 1000, 1500000), "frac": round(rng.uniform(0.1, 0.5), 3)}
    if kind == "stress":
        return {"kind": kind, "n": _log_uniform(rng, 20000, 500000), "sigma": round(rng.uniform(0.02, 0.05), 3)}
    if kind == "batch":
        return {"kind": kind, "meshes": _log_uniform(rng, 4, 96), "lo": 100, "hi": _log_uniform(rng, 3000, 100000),
                "sigma": round(rng.uniform(0.05, 0.1), 3)}
    if kind == "serve":
        return {"kind": kind, "meshes": _log_uniform(rng, 4, 48), "lo": 1000, "hi": _log_uniform(rng, 5000, 200000),
                "walkers": round(rng.uniform(0.005, 0.5), 3), "queries": _log_uniform(rng, 1000, 100000)}
    if kind == "frnn":
        return {"kind": kind, "n": _log_uniform(rng, 1000, 1500000), "r": rng.choice([1.0, 2.0, 3.0]),
                "periodic": rng.random() < 0.5, "inplace": rng.random() < 0.5}
    if kind == "rings":
        return {"kind": kind, "n": _log_uniform(rng, 1000, 600000), "row": rng.random() < 0.5}
    if kind == "build":
        return {"kind": kind, "n": _log_uniform(rng, 100, 200000)}
    return {"kind": kind, "n": _log_uniform(rng, 2000, 250000), "frac": round(rng.uniform(0.1, 0.5), 3)}


# -- inputs --------------------------------------------------------------------


def _spacing(n):
    return L / math.sqrt(n)


def _key(p):
    """Morton key of the unit cells of p: x in the even bits, y in the odd."""
    def spread(w):
        w = (w | (w << 16)) & np.uint64(0x0000FFFF0000FFFF)
        w = (w | (w << 8)) & np.uint64(0x00FF00FF00FF00FF)
        w = (w | (w << 4)) & np.uint64(0x0F0F0F0F0F0F0F0F)
        w = (w | (w << 2)) & np.uint64(0x3333333333333333)
        return (w | (w << 1)) & np.uint64(0x5555555555555555)

    c = p.astype(np.uint64)
    return spread(c[:, 0]) | (spread(c[:, 1]) << np.uint64(1))


def _points(n, rng):
    """n float32 points uniform in [0, 8192)^2, no two in one unit cell."""
    p = rng.random((n, 2), dtype=np.float32) * np.float32(L)
    while True:
        _, first = np.unique(_key(p), return_index=True)
        if len(first) == n:
            return p
        again = np.ones(n, bool)
        again[first] = False
        p[again] = rng.random((int(again.sum()), 2), dtype=np.float32) * np.float32(L)


def _in_order(p):
    return p[np.argsort(_key(p))]


def _sizes(case):
    """Sizes spread evenly over the logarithm of the range, in no order."""
    q = (np.random.default_rng(4).permutation(case["meshes"]) + 0.5) / case["meshes"]
    return (case["lo"] * (case["hi"] / case["lo"]) ** q).astype(int)


class _Addressed:
    """A device array that a mesh owns, for torch: keeps the mesh alive."""

    def __init__(self, owner, address, rows):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (rows, 2), "typestr": "<f4", "data": (address, False), "version": 2}


def _tensor(owner, address, rows):
    return torch.as_tensor(_Addressed(owner, address, rows), device="cuda")


def _vortex(q):
    """Taylor-Green velocity at unit-square positions (float64 tensor)."""
    t = 2 * math.pi
    return torch.stack([torch.sin(t * q[:, 0]) * torch.cos(t * q[:, 1]),
                        -torch.cos(t * q[:, 0]) * torch.sin(t * q[:, 1])], 1)


def _advect_moves(pos, n, frac):
    """Displacements of one advection step, float32, zero for the corners."""
    p = torch.from_numpy(pos)
    new = p[4:].double() + _vortex(p[4:].double() / L) * (frac * _spacing(n))
    new = new.clamp(0.0, float(HI)).float()
    d = torch.zeros_like(p)
    d[4:] = new - p[4:]
    return d


def _torus_inputs(case, seed):
    """Points of the torus [2L, 3L)^2 and the moves of a vortex with a drift."""
    n = case["n"]
    # the float grid at [2L, 3L) is coarser: points rounded down to it stay in
    # their own cells
    p = np.float32(2 * L) + np.floor(_points(n, np.random.default_rng(seed)) * 512) / np.float32(512)
    h = _spacing(n)
    v = _vortex((torch.from_numpy(p).double() - 2 * L) / L).numpy()
    d = ((v + np.array([0.3, -0.2])) * (case["frac"] * h / 1.4)).astype(np.float32)
    return p, d


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("walk", "stress"):
        n = case["n"]
        pts = workloads.precision_points(n, seed) if kind == "stress" else _points(n, rng)
        b = M.MeshBatch(build_mesh(pts))
        s = {"b": b, "seed": seed}
        s["sigma"] = torch.full((1,), case["sigma"] * _spacing(n), dtype=torch.float32, device="cuda")
        if case.get("near"):
            r = 2 * _spacing(n)
            k = int(L // r)
            s["r"] = r
            s["grid"] = M.GridCount2d(n, (0.0, 0.0), (L / k, L / k), (k, k))
            s["counts"] = torch.zeros(n, dtype=torch.int32, device="cuda")
            s["ids"] = torch.zeros(n * NEAR, dtype=torch.int32, device="cuda")
        s["stats"] = case.get("stats", False)
    elif kind in ("batch", "serve"):
        sizes = _sizes(case)
        b = M.MeshBatch.from_points([_points(int(n), rng) for n in sizes])
        s = {"b": b, "seed": seed}
        h = (L / np.sqrt(sizes)).astype(np.float32)
        s["sigma"] = torch.from_numpy(np.float32(case.get("sigma", 0.1)) * h).cuda()
        s["radius_host"] = 2 * h
        s["radius"] = torch.from_numpy(s["radius_host"]).cuda()
        if kind == "batch":
            s["near"] = torch.zeros(b.V * NEAR, dtype=torch.int32, device="cuda")
        else:
            s["contact"] = torch.from_numpy(h).cuda()
            s["frozen0"] = torch.from_numpy(_frozen(b.V, case["walkers"], rng)).cuda()
            s["frozen"] = s["frozen0"].clone()
            s["active"] = _active(case["meshes"], rng)
            s["verts"] = torch.from_numpy(rng.choice(b.V, min(case["queries"], b.V), replace=False)
                                          .astype(np.int32)).cuda()
            s["near"] = torch.zeros(len(s["verts"]) * NEAR, dtype=torch.int32, device="cuda")
            s["ring"] = torch.zeros(len(s["verts"]) * RING, dtype=torch.int32, device="cuda")
    elif kind in ("advect", "rings"):
        pts = _points(case["n"], rng)
        host = M.HostTriangulation()
        host.addDelaunayPoints(pts)
        s = {"dt": M.DeviceTriangulation(host), "ring": None}
        V = s["dt"].m_pos_size
        s["ring"] = torch.zeros(V * RING, dtype=torch.int32, device="cuda")
        if kind == "advect":
            # there and back: the points stay where a long run has them
            d = _advect_moves(host.m_pos, case["n"], case["frac"])
            p1 = torch.from_numpy(host.m_pos) + d
            s["moves"] = [d.cuda(), (torch.from_numpy(host.m_pos) - p1).cuda()]
            s["pos"] = torch.zeros((V, 2), dtype=torch.float32, device="cuda")
        else:
            s["closest"] = torch.zeros(V, dtype=torch.int32, device="cuda")
            s["row"] = case["row"]
        s["n"] = 0
    elif kind == "frnn":
        n = case["n"]
        r = case["r"] * _spacing(n)
        k = max(1, int(L / (r / 1.92)))
        p = _points(n, rng)
        s = {"grid": M.GridCount2d(n, (0.0, 0.0), (L / k, L / k), (k, k), periodic=case["periodic"]), "r": r}
        s["pos"] = torch.from_numpy(p).cuda()
        s["vel"] = torch.from_numpy(rng.standard_normal((n, 2)).astype(np.float32)).cuda() if case["inplace"] else None
        s["counts"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        s["ids"] = torch.zeros(n * FAR, dtype=torch.int32, device="cuda")
    elif kind == "build":
        s = {"points": _points(case["n"], rng)}
        s["ring"] = torch.zeros((case["n"] + 4) * RING, dtype=torch.int32, device="cuda")
    else:
        p, d = _torus_inputs(case, seed)
        t = M.PeriodicTriangulation(p, L)
        s = {"t": t, "n": 0, "moves": [torch.from_numpy(d).cuda(), torch.from_numpy(-d).cuda()]}
        s["ring"] = torch.zeros(t.n * RING, dtype=torch.int32, device="cuda")
        s["offsets"] = torch.zeros(t.n * RING, dtype=torch.uint8, device="cuda")
    if "b" in s:
        b = s["b"]
        s["counter"] = torch.zeros(b.count, dtype=torch.int64, device="cuda")
        s["d"] = torch.zeros((b.V, 2), dtype=torch.float32, device="cuda")
        if "ring" not in s:
            s["ring"] = torch.zeros(b.V * RING, dtype=torch.int32, device="cuda")
    s["kind"] = kind
    return s


def _frozen(V, walkers, rng):
    return (rng.random(V) >= walkers).astype(np.uint8)


def _active(meshes, rng):
    """Two overlapping halves of the meshes, stepped in turn."""
    order = rng.permutation(meshes)
    half = max(1, meshes // 2)
    return [np.sort(order[:half]).astype(np.int32), np.sort(order[-half - meshes // 8:]).astype(np.int32)]


# -- one pass ------------------------------------------------------------------


def run(s):
    kind = s["kind"]
    if kind in ("walk", "stress", "batch"):
        b = s["b"]
        b.walk(s["sigma"], s["counter"], s["d"], seed=s["seed"])
        b.settle(s["d"], sync=False)
        b.step(s["d"], stats=s.get("stats", False))
        b.one_ring(RING, s["ring"], sync=False)
        out = {"positions": _tensor(b, b.positions_ptr, b.V), "ring": s["ring"]}
        if kind == "batch":
            b.frnn_grid(s["radius_host"], s["radius"], NEAR, s["near"], sync=False)
            out["near"] = s["near"]
        elif "grid" in s:
            s["grid"].build(out["positions"][4:])
            s["grid"].frnn_ids(s["r"], NEAR, s["counts"], s["ids"], overflow=False)
            out["counts"], out["ids"] = s["counts"], s["ids"]
        return out
    if kind == "serve":
        b = s["b"]
        b.set_active(s["active"][0])
        s["active"].reverse()
        b.walk(s["sigma"], s["counter"], s["d"], seed=s["seed"], frozen=s["frozen0"])
        b.settle(s["d"], sync=False)
        b.step(s["d"], stats=False)
        s["frozen"].copy_(s["frozen0"])
        b.dla_freeze(s["contact"], s["frozen"], sync=False)
        b.frnn_list(s["radius"], s["verts"], NEAR, s["near"], sync=False)
        b.one_ring_list(s["verts"], RING, s["ring"], sync=False)
        return {"positions": _tensor(b, b.positions_ptr, b.V), "frozen": s["frozen"], "near": s["near"],
                "ring": s["ring"]}
    if kind == "advect":
        dt = s["dt"]
        dt.step(s["moves"][s["n"] & 1], stats=False)
        s["n"] += 1
        dt.oneRing(RING, s["ring"])
        return {"positions": dt.positions(out=s["pos"]), "ring": s["ring"]}
    if kind == "rings":
        dt = s["dt"]
        if s["row"]:
            dt.oneRing2(RING, s["ring"])
            dt.closestNeighbors2(RING, s["ring"], s["closest"])
        else:
            dt.oneRing(RING, s["ring"])
            dt.closestNeighbors(RING, s["ring"], s["closest"])
        return {"ring": s["ring"], "closest": s["closest"]}
    if kind == "frnn":
        g = s["grid"]
        if s["vel"] is None:
            g.build(s["pos"])
            g.frnn_ids(s["r"], FAR, s["counts"], s["ids"], overflow=False)
            return {"counts": s["counts"], "ids": s["ids"]}
        g.update(s["pos"], s["vel"])
        g.frnn(s["pos"], s["r"], FAR, s["counts"], s["ids"])
        return {"positions": s["pos"], "velocities": s["vel"], "counts": s["counts"], "ids": s["ids"]}
    if kind == "build":
        pts = s["points"].copy()
        b = M.MeshBatch(build_mesh(pts))
        b.one_ring(RING, s["ring"], sync=False)
        b.close()
        return {"points": pts, "ring": s["ring"]}
    t = s["t"]
    t.step(s["moves"][s["n"] & 1])
    s["n"] += 1
    t.oneRing(RING, s["ring"], s["offsets"])
    return {"positions": _tensor(t, t.positions_ptr(), t.n), "ring": s["ring"], "offsets": s["offsets"]}


# -- what a pass cannot do without -----------------------------------------------


def work(case):
    """Bytes: inputs read once and outputs written once.  A step reads the
    positions (8 per vertex), the displacement or the random state, and the
    edge records (16 per edge, 3 edges per vertex), writes positions; a ring
    table costs 28 per vertex and reads 52; a neighbour row 4 per neighbour.
    Operations: an incircle and two orientations per edge (40 in all), 7 per
    candidate distance."""
    kind = case["kind"]
    if kind in ("walk", "stress", "advect", "torus"):
        n = case["n"]
        by, fl = n * (24 + 48 + 28), 3 * n * 40
        if case.get("near"):
            by, fl = by + n * (8 + 4 + 4 * 12.6), fl + 7 * n * 12.6
        return {"bytes": by, "flops": fl}
    if kind in ("batch", "serve"):
        n = case["meshes"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        if kind == "batch":
            return {"bytes": n * (24 + 48 + 28 + 8 + 4 + 4 * 12.6), "flops": n * (120 + 7 * 12.6)}
        q = min(case["queries"], n)
        # the walkers of half of the meshes, their stars, every active vertex's flag and position
        return {"bytes": n * 0.5 * (1 + 8 + 8 + 8) + n * 0.5 * case["walkers"] * 12 * 16 + q * (4 + 28 + 4 * 12.6),
                "flops": n * 0.5 * case["walkers"] * 12 * 40 + q * 7 * 12.6}
    if kind == "frnn":
        n, k = case["n"], math.pi * case["r"] ** 2
        return {"bytes": n * (8 + 4 + 4 * k + (24 if case["inplace"] else 0)), "flops": 7 * n * k}
    if kind == "rings":
        return {"bytes": case["n"] * (52 + 28 + 12), "flops": case["n"] * 6 * 5}
    n = case["n"]
    return {"bytes": n * (8 + 8 + 96 + 28), "flops": 3 * n * 40}


# -- the computed numbers of the first pass in 64 bits ----------------------------


def _mix64(z):
    with np.errstate(over="ignore"):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


_CORNERS = np.array([[-1e7, -1e7], [1e7, -1e7], [1e7, 1e7], [-1e7, 1e7]])


def _walked(p, sigma, key):
    """Points (in vertex order) after the first walk step, corners first: the
    counter-based normal draws of local vertex ids 4.. under this key."""
    v = np.arange(4, 4 + len(p), dtype=np.uint64)
    a = _mix64(np.uint64(key) ^ _mix64(v))
    u1 = ((a >> np.uint64(40)).astype(np.float64) + 1.0) / 16777216.0
    u2 = ((a >> np.uint64(16)) & np.uint64(0xFFFFFF)).astype(np.float64) / 16777216.0
    rad = np.sqrt(-2.0 * np.log(u1))
    z = np.stack([rad * np.cos(2 * math.pi * u2), rad * np.sin(2 * math.pi * u2)], 1)
    return np.concatenate([_CORNERS, np.clip(p.astype(np.float64) + float(sigma) * z, 0.0, float(HI))])


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "walk":
        p = _in_order(_points(case["n"], rng))
        out = {"positions": _walked(p, np.float32(case["sigma"] * _spacing(case["n"])), seed), "ring": None}
        return dict(out, counts=None, ids=None) if case["near"] else out
    if kind in ("batch", "serve"):
        sizes = _sizes(case)
        sets = [_in_order(_points(int(n), rng)) for n in sizes]
        h = (L / np.sqrt(sizes)).astype(np.float32)
        sg = np.float32(case.get("sigma", 0.1)) * h
        new = [_walked(p, sg[c], seed + c) for c, p in enumerate(sets)]
        if kind == "batch":
            return {"positions": np.concatenate(new), "ring": None, "near": None}
        old = [np.concatenate([_CORNERS, p.astype(np.float64)]) for p in sets]
        frozen = _frozen(sum(len(p) for p in old), case["walkers"], rng)
        active = set(_active(case["meshes"], rng)[0].tolist())
        pos = np.concatenate([q if c in active else p for c, (p, q) in enumerate(zip(old, new))])
        pos[frozen != 0] = np.concatenate(old)[frozen != 0]
        return {"positions": pos, "frozen": None, "near": None, "ring": None}
    if kind == "advect":
        p = np.concatenate([_CORNERS.astype(np.float32), _in_order(_points(case["n"], rng))])
        return {"positions": p.astype(np.float64) + _advect_moves(p, case["n"], case["frac"]).double().numpy(),
                "ring": None}
    if kind == "frnn" and case["inplace"]:
        n = case["n"]
        k = max(1, int(L / (case["r"] * _spacing(n) / 1.92)))
        p = _points(n, rng)
        vel = rng.standard_normal((n, 2)).astype(np.float32)
        c = np.clip(np.floor(p / np.float32(L / k)), 0, k - 1).astype(np.int64)
        if case["periodic"]:
            c = np.floor(p / np.float32(L / k)).astype(np.int64) % k
        order = np.argsort(c[:, 1] * k + c[:, 0], kind="stable")
        return {"positions": p[order].astype(np.float64), "velocities": vel[order].astype(np.float64), "counts": None,
                "ids": None}
    if kind == "build":
        return {"points": _in_order(_points(case["n"], rng)).astype(np.float64), "ring": None}
    if kind == "torus":
        p, d = _torus_inputs(case, seed)
        q = p.astype(np.float64) + d.astype(np.float64)
        q = np.where(q >= 3 * L, q - L, np.where(q < 2 * L, q + L, q))
        return {"positions": q, "ring": None, "offsets": None}
    return None
