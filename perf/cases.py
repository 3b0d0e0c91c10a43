"""What the engine is timed on: the batched queries and loops of a transport
or ray-tracing program, through the Python front end (xdg_gb300.engine), on
the models of the benchmark and the tests.

Models (built once per process, as a program loads its geometry once):

* ``box``     an icosphere (5,120 triangles) inside a cube: volumes 1, 2 and
              the implicit complement 3;
* ``nested``  eight nested jittered icospheres, 655,360 triangles, nine
              volumes;
* ``cube``    a jittered cube of 750,000 tets;
* ``blocks``  three jittered blocks of 162,000 tets with gaps between them.

A case names the operation (``op``), its model, the number of rays, points,
tracks or particles (``n``) and the precision; ``host`` cases take NumPy arrays
and return them, the others hold device arrays.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from xdg_gb300 import synth
from xdg_gb300.engine import ANY, ENTERING, EXITING, FP64, INFTY, MIXED, XDG

PRECISION = {"mixed": MIXED, "fp64": FP64}
ORIENTATION = {"exiting": EXITING, "entering": ENTERING, "any": ANY}
DEV = "cuda:0"
CUBE_N, CUBE_SIZE = 50, 10.0     # hexes per axis (6 tets each) and edge of ``cube``
HISTORY = 16                     # faces a surface-tracking particle remembers
# room for the segments of a batch, per track (their means are 48 and 127, and
# a batch of 1,000 tracks is within 10 % of them)
CAPACITY = {"tally": 64, "segments": 192}

# ops by the model they run on, with the smallest and largest n of each
# precision that drawn cases take
RAY_OPS = ("ray_fire", "occluded", "point_in_volume", "find_volume", "closest")
RANGE = {
    "ray_fire": (1_000, 10_000_000, 3_000_000),
    "occluded": (1_000, 10_000_000, 3_000_000),
    "point_in_volume": (1_000, 10_000_000, 3_000_000),
    "find_volume": (1_000, 5_000_000, 1_000_000),
    "closest": (1_000, 1_000_000, 100_000),
    "find_element": (1_000, 5_000_000, 2_000_000),
    "next_element": (1_000, 5_000_000, 2_000_000),
    "tally": (1_000, 1_000_000, 300_000),
    "segments": (1_000, 400_000, 80_000),
    "transport_elements": (1_000, 200_000, 50_000),
    "transport_surfaces": (1_000, 200_000, 60_000),
}


def listed():
    return [
        # The smallest batch a transport code sends: the rays of one small
        # generation in a simple geometry.  Launch and latency count.
        {"name": "ray_fire_1k", "op": "ray_fire", "model": "box", "n": 1000, "precision": "mixed",
         "orientation": "exiting", "limit": False, "host": False},
        # A host code behind the plugin API: NumPy arrays in, NumPy arrays out,
        # an ordinary batch of an odd size, each ray limited to its collision
        # distance.
        {"name": "ray_fire_host_20k", "op": "ray_fire", "model": "nested", "n": 20_011,
         "precision": "mixed", "orientation": "exiting", "limit": True, "host": True},
        # The sphere-in-box configuration of the benchmark: 1e5 rays.
        {"name": "ray_fire_box_1e5", "op": "ray_fire", "model": "box", "n": 100_000,
         "precision": "mixed", "orientation": "exiting", "limit": False, "host": False},
        # The headline workload: 1e7 rays of nine volumes, each in its own.
        {"name": "ray_fire_nested_1e7", "op": "ray_fire", "model": "nested", "n": 10_000_000,
         "precision": "mixed", "orientation": "exiting", "limit": False, "host": False},
        # The plain double-precision drop-in on the same geometry.
        {"name": "ray_fire_fp64_1e6", "op": "ray_fire", "model": "nested", "n": 1_000_003,
         "precision": "fp64", "orientation": "exiting", "limit": False, "host": False},
        # Source sampling: which volume holds each point.
        {"name": "find_volume_1e6", "op": "find_volume", "model": "nested", "n": 1_000_000,
         "precision": "mixed", "orientation": "any", "limit": False, "host": False},
        # Safety distances: the nearest facet of a small and of a large batch.
        {"name": "closest_30k", "op": "closest", "model": "nested", "n": 30_011,
         "precision": "mixed", "orientation": "any", "limit": False, "host": False},
        {"name": "closest_1e6", "op": "closest", "model": "nested", "n": 1_000_000,
         "precision": "mixed", "orientation": "any", "limit": False, "host": False},
        # Track-length tallies on a mesh: locate each start, then walk.
        {"name": "tally_1e6", "op": "tally", "model": "cube", "n": 1_000_000, "precision": "mixed",
         "orientation": "any", "limit": False, "host": False},
        # The same in plain double precision, an odd and smaller batch.
        {"name": "tally_fp64_50k", "op": "tally", "model": "cube", "n": 50_021,
         "precision": "fp64", "orientation": "any", "limit": False, "host": False},
        # Tracks across meshed blocks and the gaps between them.
        {"name": "segments_100k", "op": "segments", "model": "blocks", "n": 100_000,
         "precision": "mixed", "orientation": "any", "limit": False, "host": False},
        # The surface-tracking particle loop, every event on the device.
        {"name": "particles_1e6", "op": "transport_surfaces", "model": "nested", "n": 1_000_000,
         "precision": "mixed", "orientation": "any", "limit": False, "host": False},
    ]


def draw(rng):
    op = rng.choice(sorted(RANGE))
    lo, hi, hi64 = RANGE[op]
    precision = "fp64" if rng.random() < 0.3 else "mixed"
    if precision == "fp64":
        hi = hi64
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.5:
        n |= 1
    model = {"segments": "blocks", "transport_surfaces": "nested"}.get(op, "cube")
    if op in RAY_OPS:
        model = rng.choice(["box", "nested"])
    # (host arrays for the queries a host code sends, up to what it batches)
    host = op in RAY_OPS + ("find_element", "next_element") and n <= 1_000_000 and rng.random() < 0.25
    return {"op": op, "model": model, "n": n, "precision": precision,
            "orientation": rng.choice(["exiting", "exiting", "entering", "any"])
            if op == "ray_fire" else "any",
            "limit": op == "ray_fire" and rng.random() < 0.3, "host": bool(host)}


# --------------------------------------------------------------------------
# models and inputs
# --------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _model(name):
    if name == "box":
        return synth.single_sphere_in_box(level=4)
    if name == "nested":
        return synth.nested_spheres(8, 6, 1e-3, 7)
    if name == "cube":
        tm = synth.tet_cube(CUBE_N, CUBE_SIZE, 0.2, 11)
        return synth.Model(volumes=[1], tets=tm,
                           elements={1: np.arange(len(tm.conn), dtype=np.int32)})
    return synth.tet_blocks([((12.0 * k, 0.0, 0.0), 30, 10.0) for k in range(3)], jitter=0.2,
                            seed=17)


def _uniform(g, lo, hi, n, cols=3):
    lo = torch.tensor(lo, dtype=torch.float64, device=DEV)
    hi = torch.tensor(hi, dtype=torch.float64, device=DEV)
    return lo + (hi - lo) * torch.rand((n, cols), dtype=torch.float64, device=DEV, generator=g)


def _directions(g, n):
    """Unit vectors uniform on the sphere."""
    z = 2.0 * torch.rand(n, dtype=torch.float64, device=DEV, generator=g) - 1.0
    phi = 2.0 * math.pi * torch.rand(n, dtype=torch.float64, device=DEV, generator=g)
    s = torch.sqrt((1.0 - z * z).clamp_min(0.0))
    return torch.stack([s * torch.cos(phi), s * torch.sin(phi), z], 1).contiguous()


def _exponential(g, mean, n):
    u = torch.rand(n, dtype=torch.float64, device=DEV, generator=g)
    return -mean * torch.log1p(-u)


def _inputs(case, seed):
    """The batch's own arrays, from the seed alone."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    n, model = case["n"], case["model"]
    if model in ("box", "nested"):
        # the box model's rays start inside it, those of the spheres also in
        # the implicit complement around them
        half = 19.9 if model == "box" else 9.0
        p = _uniform(g, [-half] * 3, [half] * 3, n)
        return {"p": p, "u": _directions(g, n), "limit": _exponential(g, 2.0, n)}
    if model == "cube":
        # uniform starts, isotropic directions, exponential lengths clipped at the cube
        p = _uniform(g, [0.0] * 3, [CUBE_SIZE] * 3, n)
        u = _directions(g, n)
        wall = torch.where(u > 0, CUBE_SIZE - p, -p) / u
        length = torch.minimum(_exponential(g, 5.0, n), wall.min(1).values)
        return {"p": p, "u": u, "length": length.contiguous()}
    lo, hi = [-3.0, -1.0, -1.0], [37.0, 11.0, 11.0]
    return {"p": _uniform(g, lo, hi, n), "q": _uniform(g, lo, hi, n)}


def _streams(seed, n):
    """Independent 64-bit random-stream states."""
    return torch.from_numpy(np.random.default_rng(seed).integers(-2**63, 2**63 - 1, n,
                                                                 dtype=np.int64)).to(DEV)


def prepare(case, seed):
    model = _model(case["model"])
    x = XDG(model, device=0)
    x.prepare_raytracer()
    s = _inputs(case, seed)
    n, op = case["n"], case["op"]
    s.update(case=case, x=x, precision=PRECISION[case["precision"]],
             orientation=ORIENTATION[case["orientation"]])
    if case["model"] in ("box", "nested"):
        # each ray or point belongs to the volume that holds its start
        vols = x.find_volume(s["p"], s["u"], precision=MIXED)
        lut = torch.tensor([-1] + [x.volume_to_surface_tree[v] for v in model.volumes],
                           dtype=torch.int32, device=DEV)
        s["trees"] = lut[vols.long()].contiguous()
        if op == "transport_surfaces":
            # sources outside the outer sphere start at its centre instead
            out = vols == model.implicit_complement
            s["p"][out] *= 0.2
            vols = x.find_volume(s["p"], s["u"], precision=MIXED)
            s["trees"] = lut[vols.long()].contiguous()
            s["graveyard"] = x.volume_to_surface_tree[model.implicit_complement]
            s["rng"] = _streams(seed, n)
        if not case["limit"]:
            s["limit"] = None
    if op == "segments":
        s["ipc"] = x.volume_to_surface_tree[model.implicit_complement]
    if op in ("next_element", "transport_elements"):
        s["elem"] = x.find_element(s["p"], precision=MIXED)[1]
        if op == "transport_elements":
            s["rng"] = _streams(seed, n)
    torch.cuda.synchronize()
    if case["host"]:
        for k, v in s.items():
            if isinstance(v, torch.Tensor):
                s[k] = v.cpu().numpy()
    return s


def _used(elem, length, off):
    """The segment arrays with the unused end of their capacity marked."""
    total = int(off[-1])
    elem[total:] = -1
    length[total:] = 0.0
    return elem, length


def run(state):
    s = state
    x, case, prec = s["x"], s["case"], s["precision"]
    rti, op = x.rti, case["op"]
    if op == "ray_fire":
        return rti.ray_fire(0, s["p"], s["u"], s["limit"], s["orientation"], None, prec,
                            ray_trees=s["trees"], status=True)
    if op == "occluded":
        return rti.occluded(0, s["p"], s["u"], prec, ray_trees=s["trees"])
    if op == "point_in_volume":
        return rti.point_in_volume(0, s["p"], s["u"], None, prec, ray_trees=s["trees"])
    if op == "find_volume":
        return x.find_volume(s["p"], s["u"], prec)
    if op == "closest":
        return rti.closest(0, s["p"], prec, ray_trees=s["trees"])
    if op == "find_element":
        return x.find_element(s["p"], precision=prec)
    if op == "next_element":
        return x.next_element(s["elem"], s["p"], s["u"], prec)
    if op == "tally":
        cap = CAPACITY[op] * case["n"]
        _, start = x.find_element(s["p"], precision=prec)
        elem, length, off, status = rti.walk_elements_packed(start, s["p"], s["u"], s["length"],
                                                             cap, precision=prec)
        return *_used(elem, length, off), off, status
    if op == "segments":
        cap = CAPACITY[op] * case["n"]
        elem, length, off, status = rti.segments_global(s["ipc"], rti.global_element_tree, s["p"],
                                                        s["q"], cap, precision=prec)
        return *_used(elem, length, off), off, status
    # the particle loops update their state in place: every pass starts from
    # the sources
    n = case["n"]
    pos, u, rng = s["p"].clone(), s["u"].clone(), s["rng"].clone()
    dist = torch.zeros(n, dtype=torch.float64, device=DEV)
    events = torch.zeros(n, dtype=torch.int32, device=DEV)
    if op == "transport_elements":
        elem = s["elem"].clone()
        status = rti.transport_elements(elem, pos, u, rng, 1.0, 1_000_000, dist, events,
                                        precision=prec)
        return elem, pos, u, rng, dist, events, status
    tree = s["trees"].clone()
    hist = torch.zeros((n, HISTORY), dtype=torch.int32, device=DEV)
    count = torch.zeros(n, dtype=torch.int32, device=DEV)
    status = rti.transport_surfaces(tree, pos, u, rng, 1.0, 1_000_000, hist, count, dist, events,
                                    graveyard_tree=s["graveyard"], precision=prec)
    return tree, pos, u, rng, hist, count, dist, events, status


# --------------------------------------------------------------------------
# the least work of a pass
# --------------------------------------------------------------------------

# per item: bytes read and written once (the caller's arrays), and
# floating-point operations of the exact tests that decide the outputs -- the
# Pluecker test of the hit triangle (47, a division counted as one), the
# walk's step (63 with its one face), a containment (60) or closest-point
# test (90).  Mean steps and events per item are those of the models above.
_SEGS, _BLOCK_SEGS, _EVENTS, _FLIGHTS = 48.4, 127.0, 205.0, 28.0
_WORK = {
    "ray_fire": (48 + 4 + 20, 47 + 5),
    "occluded": (48 + 4 + 12, 47),
    "point_in_volume": (48 + 4 + 4, 47 + 5),
    "find_volume": (48 + 8, 4 * (47 + 5)),
    "closest": (24 + 4 + 12, 90),
    "find_element": (24 + 8, 60),
    "next_element": (52 + 16, 56),
    "tally": (24 + 60 + 12 + 12 * _SEGS, 60 + 63 * _SEGS),
    "segments": (48 + 8 + 12 * _BLOCK_SEGS, 63 * _BLOCK_SEGS),
    "transport_elements": (2 * 72 + 4, 100 * _EVENTS),
    "transport_surfaces": (2 * (76 + 4 * HISTORY) + 4, 150 * _FLIGHTS),
}


def _model_bytes(name):
    """The geometry read once: 9 doubles a triangle, or 4 connectivity and 4
    adjacency indices a tet and its share of the vertices."""
    if name in ("box", "nested"):
        return 72 * (5132 if name == "box" else 655_360)
    return 36 * (750_000 if name == "cube" else 486_000)


def work(case):
    b, f = _WORK[case["op"]]
    b += 8 if case["limit"] else 0
    n = case["n"]
    # a small batch cannot touch the whole geometry: at most 500 bytes an item
    return {"bytes": float(b * n + min(_model_bytes(case["model"]), 500 * n)),
            "flops": float(f * n)}


# --------------------------------------------------------------------------
# the same outputs from plain torch in 64 bits
# --------------------------------------------------------------------------

PAIRS = 6_000_000_000   # brute force over at most this many (item, triangle) pairs


def _dot(a, b):
    return (a * b).sum(-1)


def _triangles(model, volume):
    """(tris [m, 3, 3], sense [m] +1 forward / -1 reverse) of a volume."""
    tris, sense = [], []
    for surf, rev in model.volume_surfaces(volume):
        t = surf.tri_xyz().reshape(-1, 3, 3)
        tris.append(t)
        sense.append(np.full(len(t), -1.0 if rev else 1.0))
    return (torch.from_numpy(np.concatenate(tris)).to(DEV),
            torch.from_numpy(np.concatenate(sense)).to(DEV))


def _first_hit(p, u, tris, sense, orientation, limit):
    """Distance to the nearest triangle hit by each ray (INFTY: none)."""
    a, e1, e2 = tris[:, 0], tris[:, 1] - tris[:, 0], tris[:, 2] - tris[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    best = torch.full((len(p),), float("inf"), dtype=torch.float64, device=DEV)
    step = max(1, 20_000_000 // len(tris))
    for k in range(0, len(p), step):
        o, d = p[k:k + step], u[k:k + step]
        # o + t d = a + b1 e1 + b2 e2 by Cramer's rule, in matrix products
        det = -(d @ nrm.T)
        na = _dot(nrm, a)
        t = (o @ nrm.T - na) / det
        m = torch.linalg.cross(d, o)
        b1 = (d @ torch.linalg.cross(a, e2).T - m @ e2.T) / det
        b2 = (m @ e1.T - d @ torch.linalg.cross(a, e1).T) / det
        ok = (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t >= 0) & torch.isfinite(t)
        along = -det * sense
        if orientation == "exiting":
            ok &= along >= 0
        elif orientation == "entering":
            ok &= along < 0
        best[k:k + step] = torch.where(ok, t, float("inf")).min(1).values
    if limit is not None:
        best = torch.where(best <= limit, best, float("inf"))
    return torch.where(torch.isfinite(best), best, INFTY)


def _nearest(p, tris):
    """Distance of each point to the nearest triangle."""
    a, b, c = tris[:, 0], tris[:, 1], tris[:, 2]
    best = torch.empty(len(p), dtype=torch.float64, device=DEV)
    step = max(1, 4_000_000 // len(tris))
    nrm = torch.linalg.cross(b - a, c - a)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    for k in range(0, len(p), step):
        q = p[k:k + step, None, :]
        d2 = torch.full((q.shape[0], len(tris)), float("inf"), dtype=torch.float64, device=DEV)
        inside = torch.ones_like(d2, dtype=torch.bool)
        for v, w in ((a, b), (b, c), (c, a)):
            e, r = w - v, q - v
            s = ((r * e).sum(-1) / _dot(e, e)).clamp(0.0, 1.0)
            d2 = torch.minimum(d2, (r - s[..., None] * e).square().sum(-1))
            inside &= (r * torch.linalg.cross(nrm, e)).sum(-1) >= 0
        h = ((q - a) * nrm).sum(-1)
        best[k:k + step] = torch.where(inside, h.square(), d2).min(1).values.sqrt()
    return best


def _locate(tm, p):
    """Tet of the jittered cube that holds each point: the one of the 27
    surrounding hexes' tets whose least barycentric coordinate is largest."""
    xyz = torch.from_numpy(tm.vertices).to(DEV)
    conn = torch.from_numpy(tm.conn.astype(np.int64)).to(DEV)
    cell = (p * (CUBE_N / CUBE_SIZE)).floor().long().clamp(0, CUBE_N - 1)
    best = torch.full((len(p),), -float("inf"), dtype=torch.float64, device=DEV)
    tet = torch.zeros(len(p), dtype=torch.int64, device=DEV)
    for i in (-1, 0, 1):
        for j in (-1, 0, 1):
            for k in (-1, 0, 1):
                c = cell + torch.tensor([i, j, k], device=DEV)
                ok = ((c >= 0) & (c < CUBE_N)).all(1)
                h = ((c[:, 0] * CUBE_N + c[:, 1]) * CUBE_N + c[:, 2]).clamp(0, CUBE_N ** 3 - 1)
                for m in range(6):
                    e = 6 * h + m
                    v = xyz[conn[e]]
                    x1, x2, x3, r = (w - v[:, 0] for w in (v[:, 1], v[:, 2], v[:, 3], p))
                    c23 = torch.linalg.cross(x2, x3)
                    det = _dot(x1, c23)
                    l1 = _dot(r, c23) / det
                    l2 = _dot(r, torch.linalg.cross(x3, x1)) / det
                    l3 = _dot(r, torch.linalg.cross(x1, x2)) / det
                    low = torch.stack([l1, l2, l3, 1 - l1 - l2 - l3]).min(0).values
                    low = torch.where(ok, low, -float("inf"))
                    better = low > best
                    best = torch.where(better, low, best)
                    tet = torch.where(better, e, tet)
    return tet


def _exit(xyz, conn, faces, tet, p, u):
    """(distance along the ray from p to the exit face of its tet, face)."""
    v = xyz[conn[tet]]                                 # [n, 4, 3]
    f = v[:, faces]                                    # [n, 4 faces, 3, 3]
    nrm = torch.linalg.cross(f[:, :, 1] - f[:, :, 0], f[:, :, 2] - f[:, :, 0])
    along = (nrm * u[:, None]).sum(-1)
    t = (nrm * (f[:, :, 0] - p[:, None])).sum(-1) / along
    return torch.where(along > 0, t, float("inf")).min(1)


def _mesh(tm):
    return (torch.from_numpy(tm.vertices).to(DEV),
            torch.from_numpy(tm.conn.astype(np.int64)).to(DEV),
            torch.from_numpy(tm.adj.astype(np.int64)).to(DEV),
            torch.from_numpy(tm.face_table.astype(np.int64)).to(DEV))


def _walk_lengths(tm, p, u, length):
    """The lengths of each track's segments, track after track."""
    xyz, conn, adj, faces = _mesh(tm)
    tet = _locate(tm, p)
    at = torch.zeros(len(p), dtype=torch.float64, device=DEV)
    ids = torch.arange(len(p), device=DEV)
    rows, lens = [], []
    while len(ids):
        t, f = _exit(xyz, conn, faces, tet, p[ids], u[ids])
        end = torch.minimum(t, length[ids])
        rows.append(ids)
        lens.append(end - at)
        nxt = adj[tet, f]
        keep = (t < length[ids]) & (nxt >= 0)
        ids, tet, at = ids[keep], nxt[keep], end[keep]
    rows, lens = torch.cat(rows), torch.cat(lens)
    return lens[torch.sort(rows, stable=True).indices]


def exact(case, seed):
    op, n = case["op"], case["n"]
    if op not in ("ray_fire", "occluded", "closest", "next_element", "tally"):
        # whole numbers; or positions that hang on every earlier rounding (a
        # particle's history, a track set back 1e-10 at each re-entry)
        return None
    model = _model(case["model"])
    if op in ("ray_fire", "occluded", "closest"):
        total = sum(len(s.face_ids) for s in model.surfaces)
        if n * (2 * total / len(model.volumes)) * (4 if op == "closest" else 1) > PAIRS:
            return None
    s = _inputs(case, seed)
    p, u = s["p"], s["u"]
    if op == "tally":
        length = torch.zeros(CAPACITY[op] * n, dtype=torch.float64, device=DEV)
        lens = _walk_lengths(model.tets, p, u, s["length"])
        length[:len(lens)] = lens
        return [None, length, None, None]
    if op == "next_element":
        xyz, conn, _, faces = _mesh(model.tets)
        return [None, _exit(xyz, conn, faces, _locate(model.tets, p), p, u).values, None]
    # the volume of each start, from the spheres' nested order: a start is
    # inside a surface when a ray along u leaves it first
    home = torch.full((n,), model.implicit_complement, dtype=torch.int64, device=DEV)
    for surf in reversed(model.surfaces):
        tris = torch.from_numpy(surf.tri_xyz().reshape(-1, 3, 3)).to(DEV)
        one = torch.ones(len(tris), dtype=torch.float64, device=DEV)
        out = _first_hit(p, u, tris, one, "exiting", None)
        into = _first_hit(p, u, tris, one, "entering", None)
        home = torch.where(out < into, surf.forward_volume, home)
    dist = torch.empty(n, dtype=torch.float64, device=DEV)
    for v in model.volumes:
        mine = torch.nonzero(home == v).flatten()
        if len(mine) == 0:
            continue
        tris, sense = _triangles(model, v)
        if op == "closest":
            dist[mine] = _nearest(p[mine], tris)
        else:
            limit = s["limit"][mine] if case["limit"] else None
            dist[mine] = _first_hit(p[mine], u[mine], tris, sense,
                                    case["orientation"] if op == "ray_fire" else "any", limit)
    if op == "occluded":
        return [None, torch.where(dist < INFTY, -INFTY, INFTY)]
    return [dist, None, None, None] if op == "ray_fire" else [dist, None]
