"""The pillbox bound that prunes the LBVH's nearest-triangle searches.

A child of an LBVH node with at most 256 leaves has, beside its box, a pillbox
that holds its triangles: centre c, unit axis n, half height h, radius r, each
of h and r with the slack 2^-17 of the coordinates' magnitude and rounded up to
16 bits.  A search whose best squared distance is `best` skips the child when
best is below (1024 Q)^2 (Q: the least, over its triangles, of twice the area x
shortest edge / longest edge^2) and the query's distance from the pillbox,
less 2^-17 of the query's magnitude, exceeds it.  That is exact only if the
reference's own f32 distance never lies below the bound there, whatever
Voronoi region its rounding picks.  These tests check that claim against the
oracle's f32 restatement of geo.rs on adversarial pairs: thin triangles, tiny
triangles far from the point (up to and beyond the reach), large coordinates,
points near the plane but far to the side, and patches of many triangles.
CPU only.
"""
import numpy as np
import pytest

import oracle

F = np.float32
SLACK, REACH = F(2.0 ** -17), F(1024)


def up16(x):
    return ((F(x).view(np.uint32).astype(np.uint64) + 0xFFFF) >> 16 << 16).astype(np.uint32).view(F)


def make_pill(tris):
    """(c, n, h, r, squared limit) of (T, 3, 3) float32 triangles, as the build forms them (float32)."""
    a, b, c = tris[:, 0], tris[:, 1], tris[:, 2]
    w = np.cross(b - a, c - a).astype(F)
    s = np.where((w @ w[0]) < 0, F(-1), F(1))
    n = (s[:, None] * w).sum(0, dtype=F)
    e = np.stack([((b - a) ** 2).sum(1), ((c - b) ** 2).sum(1), ((a - c) ** 2).sum(1)], 1).astype(F)
    same = [np.all(x == y, axis=1) for x, y in ((a, b), (b, c), (a, c))]
    proper = ~(same[0] | same[1] | same[2])
    with np.errstate(all="ignore"):
        q = np.sqrt((w * w).sum(1, dtype=F)) * np.sqrt(e.min(1)) / e.max(1)
    q = np.where(q > 0, q, F(0))
    limit = q[proper].min() if proper.any() else F(np.inf)
    nn = F(n @ n)
    with np.errstate(all="ignore"):
        n = (n / np.sqrt(nn)).astype(F)
    if not 0.99999 < n @ n < 1.00001:
        n = np.array([0, 0, 1], F)
    v = tris.reshape(-1, 3)
    ctr = (F(0.5) * (v.min(0) + v.max(0))).astype(F)
    o = ((v - ctr).astype(F) @ n).astype(F)
    ctr = (ctr + F(0.5) * (o.min() + o.max()) * n).astype(F)
    x = (v - ctr).astype(F)
    o = (x @ n).astype(F)
    r2 = np.max((x * x).sum(1, dtype=F) * F(1 + 2.0 ** -20) - o * o)
    slack = SLACK * np.abs(v).max()
    return ctr, n, up16(np.abs(o).max() + slack), up16(np.sqrt(max(r2, F(0))) * F(1.00001) + slack), (REACH * limit) ** 2


def pill_dist2(pill, p):
    ctr, n, h, r, _ = pill
    ps = (SLACK * np.abs(p).max(1)).astype(F)
    x = (p - ctr).astype(F)
    a = (x @ n).astype(F)
    l2 = np.maximum((x * x).sum(1, dtype=F) * F(1 - 2.0 ** -20) - a * a, F(0))
    da = np.maximum(np.abs(a) - (h + ps), F(0))
    dl = np.maximum(np.sqrt(l2) - (r + ps), F(0))
    return (da * da + dl * dl).astype(F)


def check(tris, pts):
    """Number of points at which the bound says something; fails where it is wrong."""
    pill = make_pill(tris)
    v = tris.reshape(-1, 3)
    d = oracle.generate_sdf(v, np.arange(len(v), dtype=np.uint32), pts, "none", "normal")
    d2 = np.minimum(np.abs(d).astype(np.float64) ** 2 * (1 + 2.0 ** -22), 3e38)  # the distance was rounded once more
    lb2 = pill_dist2(pill, pts)
    wrong = (d2 < pill[4]) & (lb2 > d2)
    assert not wrong.any(), (tris[:4], pts[wrong][:3], d2[wrong][:3], lb2[wrong][:3], pill)
    return int(((lb2 > 0) & (d2 < pill[4])).sum())


def around(rng, tri, dists):
    a, b, c = tri.astype(np.float64)
    n = np.cross(b - a, c - a)
    n /= max(np.linalg.norm(n), 1e-300)
    pts = []
    for d in dists:
        for _ in range(6):
            w = rng.dirichlet([1, 1, 1]) * rng.uniform(-0.5, 1.5, 3)
            base = w[0] * a + w[1] * b + w[2] * c
            side = rng.normal(size=3)
            side -= n * np.dot(n, side)
            side /= np.linalg.norm(side)
            edge = tri[rng.integers(3)].astype(np.float64)
            pts += [base + n * d * rng.choice([-1, 1]), base + side * d + n * d * rng.uniform(-1e-3, 1e-3),
                    base + rng.normal(size=3) * d, edge + side * 1e-3 * d + n * d]
    return np.array(pts).astype(F)


# shape: the angle at a; thin triangles have small Q and so a short reach
@pytest.mark.parametrize("scale,offset", [(1.0, 0.0), (1.0, 1e3), (1e-3, 1.0), (1e-2, 1.0), (1e-2, 30.0), (1e3, 1e5)])
@pytest.mark.parametrize("thin", [1.0, 0.1, 1e-2])
def test_one_triangle(scale, offset, thin):
    rng = np.random.default_rng(int(scale * 1e4) % 991 + int(offset) % 97 + int(1 / thin))
    said = 0
    for _ in range(60):
        a = rng.normal(size=3) * offset
        e = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        ang = thin * rng.uniform(0.2, 1.5)
        tri = np.stack([a, a + scale * rng.uniform(0.3, 1) * e[0],
                        a + scale * rng.uniform(0.3, 1) * (np.cos(ang) * e[0] + np.sin(ang) * e[1])]).astype(F)
        tri = tri[rng.permutation(3)]
        said += check(tri[None], around(rng, tri, scale * np.array([1e-3, 0.1, 1, 10, 50, 200, 600, 1e3, 1e4, 1e6])))
    assert said > 100, said  # the bound spoke (thin triangles have a short reach)


@pytest.mark.parametrize("m", [2, 9, 64, 256])
@pytest.mark.parametrize("offset", [0.0, 10.0])
def test_patches(m, offset):
    """Patches of a curved surface, windows turned over at random, some of no area."""
    rng = np.random.default_rng(m)
    said = 0
    for k in range(6):
        size = 0.02 * np.sqrt(m)
        uv = rng.uniform(-size / 2, size / 2, (m, 2))
        tris = np.empty((m, 3, 3))
        for j in range(3):
            p = uv + rng.normal(0, 0.01, (m, 2))
            tris[:, j] = np.stack([p[:, 0], p[:, 1], 0.5 * (p ** 2).sum(1) + 1e-3 * (k % 2) * rng.normal(size=m)], 1)
        rot = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        tris = (tris @ rot + rng.normal(size=3) * offset).astype(F)
        flip = rng.random(m) < 0.5
        tris[flip] = tris[flip][:, ::-1]
        flat = rng.random(m) < 0.1
        tris[flat, 1] = tris[flat, 0]
        pts = np.concatenate([around(rng, tris[i], np.array([0.01, 0.1, 0.5, 2, 10])) for i in rng.integers(0, m, 8)])
        said += check(tris, pts)
    assert said > 0, said


def test_no_area_and_far_magnitudes():
    z = np.zeros((1, 3, 3), F)
    assert check(z + F(2), np.array([[2, 2, 2], [3, 2, 2], [0, 0, 0]], F)) == 2  # a point
    seg = np.array([[[0, 0, 0], [0, 0, 0], [1, 0, 0]]], F)
    rng = np.random.default_rng(1)
    assert check(seg, rng.normal(size=(500, 3)).astype(F)) > 100
    # the smallest areas underflow: their Q is 0 and nothing is pruned
    tiny = (rng.normal(size=(1, 3, 3)) * 1e-30).astype(F)
    assert make_pill(tiny)[4] == 0
