"""Performance cases: the calls a program makes through mesh_to_sdf_b200's public entry points.

A case is a dict of plain values.  `kind` names the entry point:

* ``grid``   — ``SdfAccelerationMesh.grid_device`` (generate_grid_sdf against a resident mesh, device output),
* ``batch``  — ``grid_sdf_batch_device`` (many small grids in one job),
* ``points`` — ``SdfAccelerationMesh.query_device`` (query_sdf against a resident mesh, device arrays),
* ``call``   — ``generate_sdf`` on host arrays: mesh upload, build, query and result copy in one call,
* ``order``  — ``sort_cells_by_distance_device`` (the viewer's distance-ordered cell list).

Meshes and points are the seeded ones of ``mesh_to_sdf_b200.synth``: ``star`` (a closed, displaced icosphere with
20 * 4^subdiv triangles) and ``terrain`` (an open n x n height field as one triangle strip).  Each seed gives another
mesh and other points.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import mesh_to_sdf_b200 as m2s
from mesh_to_sdf_b200 import synth

METHODS = {
    "none_raycast": lambda: m2s.AccelerationMethod.none(m2s.SignMethod.Raycast),
    "none_normal": lambda: m2s.AccelerationMethod.none(m2s.SignMethod.Normal),
    "bvh_raycast": lambda: m2s.AccelerationMethod.bvh(m2s.SignMethod.Raycast),
    "bvh_normal": lambda: m2s.AccelerationMethod.bvh(m2s.SignMethod.Normal),
    "rtree": lambda: m2s.AccelerationMethod.rtree(),
    "rtree_bvh": lambda: m2s.AccelerationMethod.rtree_bvh(),
}
SIGNS = {"raycast": m2s.SignMethod.Raycast, "normal": m2s.SignMethod.Normal}


def listed():
    return [
        # One small grid per call, as an interactive tool or a request of a server asks for: latency and launches.
        dict(name="grid_small", kind="grid", mesh="star", detail=3, nx=32, ny=32, nz=32, sign="raycast"),
        # An ordinary grid around a mid-size mesh, edges that are no power of two, Normal sign.
        dict(name="grid_mid_normal", kind="grid", mesh="star", detail=5, nx=97, ny=110, nz=75, sign="normal"),
        # The benchmark's grid: 256^3 Raycast over an 82k-triangle closed mesh.
        dict(name="grid_large", kind="grid", mesh="star", detail=6, nx=256, ny=256, nz=256, sign="raycast"),
        # An open terrain strip of half a million triangles with the Normal sign: the largest grid.
        dict(name="grid_terrain", kind="grid", mesh="terrain", detail=512, nx=384, ny=384, nz=128, sign="normal"),
        # Many small grids in one job: asset processing.
        dict(name="batch_grids", kind="batch", count=24, sign="raycast"),
        # A few thousand points with the default method: physics or picking against a resident small mesh.
        dict(name="points_small", kind="points", mesh="star", detail=3, n=10000, method="rtree_bvh"),
        # A batch of ordinary size with the sign from the nearest normals.
        dict(name="points_normal", kind="points", mesh="star", detail=5, n=100001, method="bvh_normal"),
        # A million points with the default method: sampling a mesh for training or remeshing.
        dict(name="points_million", kind="points", mesh="star", detail=6, n=1000000, method="rtree_bvh"),
        # Four million points against a terrain, nearest triangle's sign: the largest batch.
        dict(name="points_terrain", kind="points", mesh="terrain", detail=512, n=4000000, method="rtree"),
        # Every point against every triangle: the exact method, for small sets or as a check of the others.
        dict(name="points_brute", kind="points", mesh="star", detail=6, n=65536, method="none_raycast"),
        # One call from host arrays to a host result, the crate's own form: build and query.
        dict(name="call_once", kind="call", mesh="star", detail=5, n=20000, method="rtree_bvh"),
        # The viewer's cell order of a 256^3 grid's distances.
        dict(name="cell_order", kind="order", n=256 ** 3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grid", "grid", "points", "points", "points", "batch", "call", "order"])
    if kind == "order":
        return dict(kind="order", n=_log(rng, 1000, 256 ** 3))
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(2, 24), sign=rng.choice(["raycast", "normal"]))
    if rng.random() < 0.3:
        mesh, detail = "terrain", _log(rng, 48, 512)
    else:
        mesh, detail = "star", rng.randint(2, 6)
    if kind == "grid":
        base = _log(rng, 16, 256)
        edges = [max(8, min(256, int(round(base * rng.uniform(0.6, 1.4))))) for _ in range(3)]
        return dict(kind="grid", mesh=mesh, detail=detail, nx=edges[0], ny=edges[1], nz=edges[2],
                    sign=rng.choice(["raycast", "normal"]) if mesh == "star" else "normal")
    if kind == "call":
        return dict(kind="call", mesh=mesh, detail=detail, n=_log(rng, 100, 100000),
                    method=rng.choice(["rtree_bvh", "bvh_normal", "rtree", "bvh_raycast"]))
    method = rng.choice(["rtree_bvh", "rtree_bvh", "rtree", "bvh_raycast", "bvh_normal", "none_raycast", "none_normal"])
    n = _log(rng, 100, 1000000)
    if method.startswith("none"):
        n = min(n, 65536, int((5.3e9 if method == "none_raycast" else 2e9) // _triangles(mesh, detail)))
    return dict(kind="points", mesh=mesh, detail=detail, n=max(100, n), method=method)


def _batch_edges(count):
    """Every edge of the batched-grid workload in turn (the meshes are drawn)."""
    return [synth.BATCH_EDGES[k % len(synth.BATCH_EDGES)] for k in range(count)]


def _triangles(mesh, detail):
    return 20 * 4 ** detail if mesh == "star" else 2 * (detail - 1) ** 2 + 4 * (detail - 2)


def _vertices(mesh, detail):
    return 10 * 4 ** detail + 2 if mesh == "star" else detail * detail


def _mesh(case, seed):
    """(vertices, Topology, (T, 3) vertex indices)."""
    if case["mesh"] == "star":
        v, idx = synth.star(case["detail"], seed)
        return v, m2s.Topology.TriangleList(idx), idx.reshape(-1, 3)
    v, idx = synth.terrain(case["detail"], seed)
    return v, m2s.Topology.TriangleStrip(idx), np.stack([idx[:-2], idx[1:-1], idx[2:]], 1)


def _box(case, v):
    """What a program samples: the mesh's box with a margin (a terrain also well above and below it)."""
    lo, hi = synth.padded_bbox(v)
    if case["mesh"] == "terrain":
        lo[2], hi[2] = -0.3, 0.5
    return lo, hi


def _queries(case, v, tri, seed):
    if case["mesh"] == "star":  # four fifths anywhere in the box, one fifth near the surface
        return synth.mixed_points(v, tri.reshape(-1), case["n"], seed + 7)
    lo, hi = _box(case, v)
    return synth.uniform_points(case["n"], lo, hi, seed + 7)


def _grid(case, v):
    lo, hi = _box(case, v)
    return m2s.Grid.from_bounding_box(lo, hi, [case["nx"], case["ny"], case["nz"]])


def _stream():
    return torch.cuda.current_stream().cuda_stream


def prepare(case, seed):
    kind = case["kind"]
    if kind == "order":
        d = _distances(case["n"], seed).cuda()
        return dict(kind=kind, d=d, order=torch.empty(case["n"], dtype=torch.int32, device="cuda"),
                    minmax=torch.empty(2, device="cuda"))
    if kind == "batch":
        meshes, grids = [], []
        edges = _batch_edges(case["count"])
        for edge, (v, idx, lo, hi, _) in zip(edges, synth.batch_meshes(case["count"], seed)):
            meshes.append(m2s.build_sdf_acceleration(v, m2s.Topology.TriangleList(idx)))
            grids.append(m2s.Grid.from_bounding_box(lo, hi, [edge] * 3))
        return dict(kind=kind, meshes=meshes, grids=grids, sign=SIGNS[case["sign"]],
                    out=torch.empty(int(m2s.grid_offsets(grids)[-1]), device="cuda"))
    v, topology, tri = _mesh(case, seed)
    if kind == "call":
        return dict(kind=kind, v=v, topology=topology, q=_queries(case, v, tri, seed), method=METHODS[case["method"]]())
    if kind == "points":
        mesh = m2s.build_sdf_acceleration(v, topology, METHODS[case["method"]]())
        q = torch.from_numpy(_queries(case, v, tri, seed)).cuda()
        return dict(kind=kind, mesh=mesh, q=q, out=torch.empty(case["n"], device="cuda"))
    mesh = m2s.build_sdf_acceleration(v, topology)
    grid = _grid(case, v)
    return dict(kind=kind, mesh=mesh, grid=grid, sign=SIGNS[case["sign"]],
                out=torch.empty(grid.get_total_cell_count(), device="cuda"))


def run(state):
    kind = state["kind"]
    if kind == "grid":
        state["mesh"].grid_device(state["grid"], state["sign"], state["out"], stream=_stream())
        return state["out"]
    if kind == "batch":
        m2s.grid_sdf_batch_device(state["meshes"], state["grids"], state["sign"], state["out"], stream=_stream())
        return state["out"]
    if kind == "points":
        state["mesh"].query_device(state["q"], state["out"], stream=_stream())
        return state["out"]
    if kind == "call":
        return m2s.generate_sdf(state["v"], state["topology"], state["q"], state["method"])
    m2s.sort_cells_by_distance_device(state["d"], state["order"], state["minmax"], stream=_stream())
    return state["order"], state["minmax"]


# Operations of the reference's f32 arithmetic: one closest point and distance; one aligned ray test; one distance of
# a point to a plane.
_CLOSEST, _RAY, _PLANE = 76, 18, 6


def work(case):
    """Inputs once, outputs once; a closest point per output (a grid cell or query has to evaluate its own nearest
    triangle), and for the method that looks at every pair a ray test (Raycast) or plane distance (Normal) per pair."""
    kind = case["kind"]
    if kind == "order":
        return {"bytes": 8 * case["n"], "flops": 0}
    if kind == "batch":  # the subdivisions are drawn: their mean
        cells = sum(e ** 3 for e in _batch_edges(case["count"]))
        tris = case["count"] * sum(20 * 4 ** s for s in synth.BATCH_SUBDIVS) / len(synth.BATCH_SUBDIVS)
        return {"bytes": int(4 * cells + 18 * tris), "flops": int(cells * _CLOSEST)}
    T, V = _triangles(case["mesh"], case["detail"]), _vertices(case["mesh"], case["detail"])
    mesh = 12 * V + (12 * T if case["mesh"] == "star" else 4 * (T + 2))
    if kind == "grid":
        cells = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": mesh + 4 * cells, "flops": cells * _CLOSEST}
    flops = case["n"] * _CLOSEST
    if case["method"].startswith("none"):
        flops += case["n"] * T * (_RAY if case["method"] == "none_raycast" else _PLANE)
    return {"bytes": mesh + 16 * case["n"], "flops": flops}


def _distances(n, seed):
    """Distances of an n-cell grid in the order a grid call gives them: a bumpy sphere's."""
    g = torch.Generator().manual_seed(seed)
    f, ph, amp = torch.rand(3, generator=g) * 5 + 1, torch.rand(3, generator=g) * 6.28, 0.1 * torch.rand(1, generator=g)
    edge = max(1, round(n ** (1 / 3)))
    i = torch.arange(n, dtype=torch.int64)
    c = [(i // (edge * edge)).float(), ((i // edge) % edge).float(), (i % edge).float()]
    c = [x * (2.4 / edge) - 1.2 for x in c]
    r = (c[0] * c[0] + c[1] * c[1] + c[2] * c[2]).sqrt()
    bumps = torch.sin(f[0] * c[0] + ph[0]) * torch.sin(f[1] * c[1] + ph[1]) + torch.sin(f[2] * c[2] + ph[2])
    return r - 1 - amp * bumps


# ---- what the outputs are in 64 bits ---------------------------------------------------------------------------

_EXACT_PAIRS = 6_000_000_000  # about a dozen seconds on the device


def _exact_points(p, tris, rule, device):
    """Signed distances of points to triangles, every pair, in 64 bits.  `rule`: "vote", inside when two of the three
    rays along +x, +y, +z cross the mesh an odd number of times; "ray", when the +x ray alone does; "first", the side of
    the nearest triangle, of several at one distance the first; "any", the same but positive if any of them (within the
    crate's 1e-6) is."""
    tris = torch.from_numpy(tris).to(device)
    a, b, c = tris[:, 0], tris[:, 1], tris[:, 2]
    area = torch.linalg.cross(b - a, c - a)
    out = np.empty(len(p))
    step = max(1, 40_000_000 // max(1, len(tris)))
    for k in range(0, len(p), step):
        q = torch.from_numpy(p[k:k + step]).to(device)[:, None, :]
        d2, side = _closest(q, a, b, c, area, rule in ("first", "any"))
        d = d2.min(1).values.sqrt()
        if rule == "ray":
            d = torch.where((_crossings(q, tris, 0) & 1) > 0, -d, d)
        elif rule == "vote":
            odd = sum((_crossings(q, tris, ax) & 1) for ax in range(3))
            d = torch.where(odd >= 2, -d, d)
        elif rule == "first":
            first = (d2.sqrt() <= d[:, None] * (1 + 1e-12) + 1e-14).to(torch.uint8).argmax(1)
            d = torch.where(side.gather(1, first[:, None])[:, 0], d, -d)
        else:
            near = d2.sqrt() <= d[:, None] + 1e-6
            d = torch.where((near & side).any(1), d, -d)
        out[k:k + step] = d.cpu().numpy()
    return out


def _dot(u, v):
    return u[..., 0] * v[..., 0] + u[..., 1] * v[..., 1] + u[..., 2] * v[..., 2]


def _closest(q, a, b, c, area, want_side):
    """Squared distance and side of every (point, triangle): the least over the three edges and, where the point lies
    over the triangle, the plane."""
    best = torch.full((q.shape[0], a.shape[0]), math.inf, dtype=torch.float64, device=a.device)
    side = torch.zeros_like(best, dtype=torch.bool)
    over = torch.ones_like(side)
    for s, e in ((a, b), (b, c), (c, a)):
        u, w = e - s, q - s
        t = (_dot(w, u) / _dot(u, u).clamp_min(1e-300)).clamp(0, 1)
        x = w - t[..., None] * u
        d2 = _dot(x, x)
        if want_side:
            side = torch.where(d2 < best, _dot(x, area) > 0, side)
        best = torch.minimum(best, d2)
        over &= _dot(torch.linalg.cross(area, u), w) >= 0
    nn = _dot(area, area)
    h = _dot(q - a, area)
    over &= nn > 0
    if want_side:
        side = torch.where(over, h > 0, side)
    return torch.where(over, torch.minimum(best, h * h / nn.clamp_min(1e-300)), best), side


def _crossings(q, tris, ax):
    y, z = (ax + 1) % 3, (ax + 2) % 3
    v = [tris[:, i] for i in range(3)]
    w = []
    for i in range(3):
        s, e = v[i], v[(i + 1) % 3]
        w.append((q[..., z] - s[:, z]) * (e[:, y] - s[:, y]) - (q[..., y] - s[:, y]) * (e[:, z] - s[:, z]))
    hit = ((w[0] > 0) & (w[1] > 0) & (w[2] > 0)) | ((w[0] < 0) & (w[1] < 0) & (w[2] < 0))
    s = w[0] + w[1] + w[2]
    x = (w[1] * v[0][:, ax] + w[2] * v[1][:, ax] + w[0] * v[2][:, ax]) / torch.where(s == 0, torch.ones_like(s), s)
    return (hit & (x > q[..., ax])).sum(1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "order":
        d = _distances(case["n"], seed)
        return None, np.array([d.min().item(), d.max().item()], np.float64)  # the order is whole numbers
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "batch":
        return None  # 24 grids against their meshes: far over the time
    v, _, tri = _mesh(case, seed)
    n = case["nx"] * case["ny"] * case["nz"] if kind == "grid" else case["n"]
    if n * len(tri) > _EXACT_PAIRS:
        return None
    if kind == "grid":
        g = _grid(case, v)
        ax = [np.float64(g.first_cell[i]) + np.arange(g.cell_count[i]) * np.float64(g.cell_size[i]) for i in range(3)]
        p = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
        rule = "vote" if case["sign"] == "raycast" else "any"
    else:
        p = _queries(case, v, tri, seed).astype(np.float64)
        rules = {"rtree": "first", "bvh_normal": "any", "none_normal": "any", "none_raycast": "ray"}
        rule = rules.get(case["method"], "vote")
    return _exact_points(p, v.astype(np.float64)[tri], rule, device)
