"""Searches over meshes of needles among ordinary triangles, bit for bit against the oracle: shapes around the one from
which a triangle has no reach (64 : 1), tiny and huge coordinates, points a few slacks outside long edges and tips."""
import numpy as np
import pytest

import mesh_to_sdf_b200 as m2s
import test_tri_reach as reach

pytestmark = pytest.mark.gpu
A, S, T = m2s.AccelerationMethod, m2s.SignMethod, m2s.Topology
METHODS = {"rtree": ("rtree", "normal", A.rtree()), "rtree_bvh": ("rtree_bvh", "raycast", A.rtree_bvh()),
           "bvh_normal": ("bvh", "normal", A.bvh(S.Normal)), "none_raycast": ("none", "raycast", A.none(S.Raycast))}


@pytest.mark.parametrize("method", list(METHODS))
@pytest.mark.parametrize("aspect,scale", [(30, 1.0), (64, 1.0), (66, 1.0), (1000, 1.0), (10000, 1.0), (64, 2.0 ** -20),
                                          (30, 2.0 ** 20)])
def test_needles(orc, aspect, scale, method):
    rng = np.random.default_rng(aspect)
    tris = np.concatenate([reach.patch(rng, 64, aspect) for _ in range(20)]) * np.float32(scale)
    v = tris.reshape(-1, 3)
    idx = np.arange(len(v), dtype=np.uint32)
    near = reach.outside_edges(rng, tris, 6000)
    q = np.concatenate([near, rng.normal(size=(3000, 3)).astype(np.float32) * np.float32(scale)]).astype(np.float32)
    accel, sign, am = METHODS[method]
    got = m2s.generate_sdf(v, T.TriangleList(idx), q, am)
    exp = orc.generate_sdf(v, idx, q, accel, sign)
    assert np.array_equal(got.view(np.uint32), exp.view(np.uint32))
