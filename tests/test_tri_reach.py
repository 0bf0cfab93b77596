"""Up to which distance the pillbox and disc bounds prune: the rule of m2s_reach.cuh, compiled here for the host.

The header's argument has two parts that can be checked on their own: how far outside a triangle the foot of the
perpendicular may lie where the reference's f32 region tests still give the face region (g below), and that within the
reach the reference's distance falls short of the true one by less than the bounds' slack.  The points are those where
rounding decides: beside vertices and edges, near the plane, at distances from far below the edges to beyond the reach;
the triangles fat, needles, caps and right-angled ones, up to and beyond the shape from which the reach is 0.  CPU only.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle
import test_pill_bound as pills

F = np.float32
U, SLACK, THIN = 2.0 ** -24, 2.0 ** -17, 64.0
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mesh_to_sdf_b200", "csrc")


@pytest.fixture(scope="module")
def tri_reach(tmp_path_factory):
    d = tmp_path_factory.mktemp("reach")
    (d / "r.cpp").write_text('#include "m2s_reach.cuh"\nextern "C" float reach(const float* t) '
                             "{ return m2s::tri_reach(t, t + 3, t + 6); }\n")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "r.so"),
                    str(d / "r.cpp")], check=True)
    fn = ctypes.CDLL(str(d / "r.so")).reach
    fn.restype = ctypes.c_float

    def call(tri):
        t = np.ascontiguousarray(tri, F)
        return float(fn(t.ctypes.data_as(ctypes.c_void_p)))

    return call


def shape(tri):
    """(longest, shortest edge, twice the area, a, Q) in 64 bits."""
    t = tri.astype(np.float64)
    e = [np.linalg.norm(t[1] - t[0]), np.linalg.norm(t[2] - t[1]), np.linalg.norm(t[0] - t[2])]
    w = np.linalg.norm(np.cross(t[1] - t[0], t[2] - t[0]))
    return max(e), min(e), w, max(e) ** 2 / w, w * min(e) / max(e) ** 2


def random_triangle(rng, most):
    thin = 1 / most ** rng.uniform(0, 1)
    x = rng.choice([rng.uniform(-0.1, 1.1), rng.choice([0, 1]) + rng.normal() * 3 * thin, rng.choice([0, 1]),
                    rng.uniform(0.3, 0.7)])
    t = np.array([[0, 0, 0], [1, 0, 0], [x, thin, 0]])
    t = (t - t.mean(0)) @ np.linalg.qr(rng.normal(size=(3, 3)))[0]
    return (t + rng.choice([0, 0, 0.3, 10]) * rng.normal(size=3)).astype(F)[rng.permutation(3)]


def points(rng, tri, n, far):
    """n points, most of them beside vertices and edges, at log-spread distances up to `far`."""
    t = tri.astype(np.float64)
    w = rng.dirichlet([1, 1, 1], n)
    i = np.arange(n)
    w[i, rng.integers(0, 3, n)] *= rng.choice([0, 1e-3, -1e-3, 1], n)
    at = np.zeros((n, 3))
    at[i, rng.integers(0, 3, n)] = 1
    lam = np.where(rng.random(n) < 0.3, 0, 10 ** rng.uniform(-6, 0, n))
    w = np.where((rng.random(n) < 0.6)[:, None], at * (1 - lam[:, None]) + w * lam[:, None], w)
    base = (w / w.sum(1, keepdims=True)) @ t
    nn = np.cross(t[1] - t[0], t[2] - t[0])
    nn /= np.linalg.norm(nn)
    side = rng.normal(size=(n, 3))
    side += (side @ nn)[:, None] * nn * (rng.choice([0, 1e-3, 0.1, 1, 10, 1e3, 1e5, 1e6, 1e7], n) - 1)[:, None]
    side /= np.linalg.norm(side, axis=1, keepdims=True)
    return (base + side * (far * 10 ** rng.uniform(-7, 0, n))[:, None]).astype(F)


def exact(tri, p):
    """Distance to the triangle and the in-plane distance of the foot from it, in 64 bits."""
    t, p = tri.astype(np.longdouble), p.astype(np.longdouble)
    nn = np.cross(t[1] - t[0], t[2] - t[0])
    nn /= np.sqrt((nn * nn).sum())
    h = (p - t[0]) @ nn
    foot = p - h[:, None] * nn
    g2 = np.full(len(p), np.inf, np.longdouble)
    over = np.ones(len(p), bool)
    for s, e in ((t[0], t[1]), (t[1], t[2]), (t[2], t[0])):
        u, w = e - s, foot - s
        x = w - np.clip(w @ u / (u @ u), 0, 1)[:, None] * u
        g2 = np.minimum(g2, (x * x).sum(1))
        over &= np.cross(nn, u) @ w.T >= 0
    g2 = np.where(over, 0, g2)
    return np.sqrt(h * h + g2), np.sqrt(g2)


def face_region(tri, p):
    """Whether closest_point_proper (geo.rs:70-138, f32) reaches its face region, and there with a weight below 0."""
    a, b, c = tri
    dot = lambda u, v: (u[..., 0] * v[..., 0] + u[..., 1] * v[..., 1]) + u[..., 2] * v[..., 2]
    ab, ac, ap, bp, cp = b - a, c - a, p - a, p - b, p - c
    d1, d2, d3, d4, d5, d6 = dot(ab, ap), dot(ac, ap), dot(ab, bp), dot(ac, bp), dot(ab, cp), dot(ac, cp)
    vc, vb, va = d1 * d4 - d3 * d2, d5 * d2 - d1 * d6, d3 * d6 - d5 * d4
    done = ((d1 <= 0) & (d2 <= 0)) | ((d3 >= 0) & (d4 <= d3)) | ((d6 >= 0) & (d5 <= d6))
    done |= ((vc <= 0) & (d1 >= 0) & (d3 <= 0)) | ((vb <= 0) & (d2 >= 0) & (d6 <= 0))
    done |= (va <= 0) & (d4 - d3 >= 0) & (d5 - d6 >= 0)
    return ~done, ~done & ((va < 0) | (vb < 0) | (vc < 0))


def reference(tri, p):
    d = oracle.generate_sdf(tri.reshape(-1, 3), np.arange(3, dtype=np.uint32), p, "none", "normal")
    return np.abs(d).astype(np.float64)


@pytest.mark.parametrize("most", [4, 64, 64, 2000])
def test_foot_and_distance(tri_reach, most):
    rng = np.random.default_rng(most)
    outside = held = 0
    for k in range(150):
        tri = random_triangle(rng, most)
        L, s, w, a, Q = shape(tri)
        reach = tri_reach(tri)
        if a > THIN * 1.001:
            assert reach == 0.0  # not covered by the argument
        if a < THIN * 0.999:
            assert abs(reach / (1024 * Q) - 1) < 1e-3
        p = points(rng, tri, 4000, 1024 * Q * rng.choice([1.01, 1.01, 300]))
        D, g = exact(tri, p)
        face, below = face_region(tri, p)
        rounding = 4 * U * (np.abs(tri).max() + np.abs(p).max(1))  # p itself is exact; the foot's own evaluation is not
        assert (g[face] <= 28 * U * (D[face] + L) ** 2 / Q + rounding[face]).all()
        if a <= THIN:
            near = below & (D <= 8 * L)
            assert (g[near] <= 28 * U * D[near] * (1.15 * D[near] / Q + a) + 19 * U * a * D[near] + rounding[near]).all()
        outside += int((face & (g > rounding)).sum())
        if reach > 0:
            r = reference(tri, p)
            slack = SLACK * (np.abs(tri).max() + np.abs(p).max(1).astype(np.float64))
            short = (D - r <= slack) | ((D > 1.01 * reach) & (r > reach))
            assert short.all(), (tri, p[~short][:3], D[~short][:3], r[~short][:3])
            held += int((D < reach).sum())
    assert held > 10000 or most > 1000, held
    assert outside > 0, outside  # feet outside the triangle; none with a weight below 0 as well was ever seen


def test_written_formula_is_not_enough(tri_reach):
    """Why the rule has more than 1024 Q: the foot's offset grows with the distance from the vertices, not from the
    triangle, so 24 u D^2 / Q (with D alone) does not bound how far outside a triangle the face region is given."""
    rng = np.random.default_rng(5)
    most = 0.0
    for _ in range(200):
        tri = random_triangle(rng, 2000)
        L, s, w, a, Q = shape(tri)
        p = points(rng, tri, 4000, 1024 * Q)
        D, g = exact(tri, p)
        face, _ = face_region(tri, p)
        if face.any():
            most = max(most, float((g[face] / (24 * U * D[face] ** 2 / Q)).max()))
    assert most > 2.0, most


def test_no_area_large_and_tiny(tri_reach):
    t = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], F)
    assert tri_reach(t) > 400
    assert tri_reach(t * F(2.0 ** -27)) == 0.0  # an area below 2^-51
    assert tri_reach(t * F(2.0 ** -24)) > 0.0
    big = t * F(2.0 ** 27)
    assert 0 < tri_reach(big) * 2.0 ** 27.5 <= 2.0 ** 52 * 1.001
    for bad in (np.nan, np.inf):
        x = t.copy()
        x[1, 0] = bad
        assert tri_reach(x) == 0.0


def patch(rng, m, aspect):
    """m ordinary triangles of a gently curved surface and needles of `aspect` among them at any tilt."""
    uv = rng.uniform(-0.1, 0.1, (m, 2))
    tris = np.empty((m, 3, 3))
    for j in range(3):
        q = uv + rng.normal(0, 0.02, (m, 2))
        tris[:, j] = np.stack([q[:, 0], q[:, 1], 0.3 * (q ** 2).sum(1)], 1)
    k = max(1, m // 3)
    d, e = rng.normal(size=(2, k, 3))
    d *= 0.05 / np.linalg.norm(d, axis=1, keepdims=True)
    e -= d * ((e * d).sum(1) / (d * d).sum(1))[:, None]
    e *= 0.1 / aspect / np.linalg.norm(e, axis=1, keepdims=True)
    mid = np.concatenate([uv[:k], rng.normal(0, 0.005, (k, 1))], 1)
    tris[:k] = np.stack([mid - d, mid + d, mid + rng.uniform(-1, 1, (k, 1)) * d + e], 1)
    return (tris @ np.linalg.qr(rng.normal(size=(3, 3)))[0] + rng.choice([0, 1]) * rng.normal(size=3)).astype(F)


def outside_edges(rng, tris, n):
    """Points a few slacks outside edges and tips, in and near the triangles' planes."""
    t = tris[rng.integers(0, len(tris), n)].astype(np.float64)
    nn = np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    nn /= np.linalg.norm(nn, axis=1, keepdims=True)
    lam = np.where(rng.random(n) < 0.5, rng.choice([0.0, 1.0], n), rng.random(n))[:, None]
    i = rng.integers(0, 3, n)
    s, e = t[np.arange(n), i], t[np.arange(n), (i + 1) % 3]
    out = -np.cross(nn, e - s)
    out /= np.maximum(np.linalg.norm(out, axis=1, keepdims=True), 1e-30)
    far = (SLACK * np.abs(tris).max() * 10 ** rng.uniform(-1, 3, n))[:, None]
    return (s + lam * (e - s) + far * (out + nn * rng.choice([0, 0.01, 1, -1], n)[:, None] + 0.3 * rng.normal(size=(n, 3)))).astype(F)


@pytest.mark.parametrize("aspect", [30, 100, 1000, 10000])
@pytest.mark.parametrize("m", [2, 9, 64])
def test_patches_with_needles(tri_reach, aspect, m):
    """The pillbox over needles and ordinary triangles, its limit from the compiled rule, against the oracle's distance."""
    rng = np.random.default_rng(aspect + m)
    for _ in range(12):
        tris = patch(rng, m, aspect)
        c, n, h, r, _ = pills.make_pill(tris)
        limit = min(tri_reach(t) for t in tris)
        v = tris.reshape(-1, 3)
        p = np.concatenate([outside_edges(rng, tris, 3000), points(rng, tris[0], 1000, 0.5)])
        d = np.abs(oracle.generate_sdf(v, np.arange(len(v), dtype=np.uint32), p, "none", "normal")).astype(np.float64)
        lb = np.sqrt(pills.pill_dist2((c, n, h, r, 0), p).astype(np.float64))
        wrong = (d < limit) & (lb > d * (1 + 2.0 ** -22))
        assert not wrong.any(), (tris, p[wrong][:3], d[wrong][:3], lb[wrong][:3])
        if aspect >= 1000:
            assert limit == 0.0  # the needles' own reach


def disc_bound2(tri, p):
    """The disc's bound as the brute-force kernel forms it (float32): squared bound."""
    t = tri.astype(F)
    w = np.cross(t[1] - t[0], t[2] - t[0]).astype(F)
    n = (w / np.sqrt(w @ w)).astype(F) * F(1 - 2.0 ** -13)
    c = ((t[0] + t[1] + t[2]) * F(1 / 3)).astype(F)
    slack = F(SLACK) * np.abs(t).max()
    radius = np.sqrt(max(((x - c) ** 2).sum() for x in t)) * F(1.00001) + slack
    ps = (F(SLACK) * np.abs(p).max(1)).astype(F)
    x = (p - c).astype(F)
    a1 = (x @ n).astype(F)
    up = a1 * F(1 + 2.0 ** -12)
    l = np.sqrt(np.maximum((x * x).sum(1, dtype=F) * F(1 - 2.0 ** -20) - up * up, F(0)))
    da, dl = np.maximum(np.abs(a1) - (slack + ps), F(0)), np.maximum(l - (radius + ps), F(0))
    return (da * da + dl * dl).astype(F)


def test_single_triangle_disc(tri_reach):
    """A disc skips its triangle when bound^2 > best^2, best < reach and bound^2 < 2^17 reach^2: never below r."""
    rng = np.random.default_rng(11)
    said = far = 0
    for _ in range(250):
        tri = random_triangle(rng, 64)
        reach = tri_reach(tri)
        ab, ac = (tri[1] - tri[0]).astype(np.float64), (tri[2] - tri[0]).astype(np.float64)
        w = np.cross(ab, ac)
        if reach == 0 or 200 * (w @ w) < (ab @ ab) * (ac @ ac) * 1.001:
            continue
        p = points(rng, tri, 3000, reach * rng.choice([1, 400]))
        r = reference(tri, p)
        lb = np.sqrt(disc_bound2(tri, p).astype(np.float64))
        used = lb * lb < 2.0 ** 17 * reach * reach
        wrong = used & (np.minimum(lb, reach) > r * (1 + 2.0 ** -22))  # some best distance between r and the bound
        assert not wrong.any(), (tri, p[wrong][:3], r[wrong][:3], lb[wrong][:3])
        said += int((used & (lb > 0)).sum())
        far += int((used & (lb > 10 * reach)).sum())
    assert said > 10000 and far > 1000, (said, far)
