"""Nearest-triangle searches with pillbox bounds, bit for bit against the oracle.

Leaf counts around the bound's own edges (8: one lane builds it, 9 to 256: a
warp, above: none) and query counts around the paths' (one warp per query up
to 10,240, on a large mesh 4,096; 2^17: Morton order, warps that start together)."""
import numpy as np
import pytest

import mesh_to_sdf_b200 as m2s
from mesh_to_sdf_b200 import synth

pytestmark = pytest.mark.gpu
A, S, T = m2s.AccelerationMethod, m2s.SignMethod, m2s.Topology
METHODS = {"rtree": ("rtree", "normal", A.rtree()), "rtree_bvh": ("rtree_bvh", "raycast", A.rtree_bvh()),
           "bvh_normal": ("bvh", "normal", A.bvh(S.Normal))}


def check(orc, v, idx, q, method, strip=False):
    accel, sign, am = METHODS[method]
    topo = T.TriangleStrip(idx) if strip else T.TriangleList(idx)
    got = m2s.generate_sdf(v, topo, q, am)
    exp = orc.generate_sdf(v, idx, q, accel, sign, strip=strip)
    bad = np.nonzero(got.view(np.uint32) != exp.view(np.uint32))[0]
    assert len(bad) == 0, (method, len(bad), q[bad[:3]], got[bad[:3]], exp[bad[:3]])


@pytest.mark.parametrize("method", list(METHODS))
@pytest.mark.parametrize("tris", [2, 3, 8, 9, 17, 256, 257, 513, 1000])
def test_leaf_counts(orc, tris, method):
    v, idx = synth.star(4, seed=3)
    rng = np.random.default_rng(tris)
    keep = idx.reshape(-1, 3)[np.sort(rng.permutation(len(idx) // 3)[:tris])].reshape(-1)
    q = synth.mixed_points(v, idx, 3000, seed=5)
    check(orc, v, keep, np.concatenate([q, 4 * q[:500]]), method)


@pytest.mark.parametrize("method", list(METHODS))
@pytest.mark.parametrize("subdiv,n", [(5, 10240), (5, 10241), (6, 4096), (6, 4097), (5, (1 << 17) - 1), (5, 1 << 17),
                                      (5, (1 << 17) + 33)])
def test_query_counts(orc, subdiv, n, method):
    v, idx = synth.star(subdiv, seed=2)
    check(orc, v, idx, synth.mixed_points(v, idx, n, seed=n % 1000), method)


@pytest.mark.parametrize("method", list(METHODS))
def test_flat_thin_and_strip(orc, method):
    # a box's large flat faces; needles; a strip with joining windows and turned windows
    rng = np.random.default_rng(3)
    cube = np.array([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)], np.float32)
    faces = np.array([0, 1, 3, 0, 3, 2, 4, 6, 7, 4, 7, 5, 0, 4, 5, 0, 5, 1, 2, 3, 7, 2, 7, 6, 0, 2, 6, 0, 6, 4, 1, 5, 7,
                      1, 7, 3], np.uint32)
    q = rng.uniform(-3, 3, (2000, 3)).astype(np.float32)
    check(orc, cube, faces, q, method)
    c = rng.normal(size=(1500, 3))
    d = rng.normal(size=(1500, 3)) * 0.2
    needles = np.stack([c + d, c - d, c + rng.normal(size=(1500, 3)) * 1e-4], 1).reshape(-1, 3).astype(np.float32)
    check(orc, needles, np.arange(len(needles), dtype=np.uint32), q, method)
    v, idx = synth.terrain(40, seed=2)
    check(orc, v, idx, rng.uniform([-0.2, -0.2, -0.3], [1.2, 1.2, 0.5], (20000, 3)).astype(np.float32), method, True)
