"""generate_sdf around the number of queries from which its tree gets pillboxes (one per 512
triangles and 2^22 pairs, for Bvh(Normal) one per 1,024 and 2^20), bit for bit."""
import numpy as np
import pytest

import mesh_to_sdf_b200 as m2s
from mesh_to_sdf_b200 import synth

pytestmark = pytest.mark.gpu
A, S = m2s.AccelerationMethod, m2s.SignMethod


@pytest.mark.parametrize("n", [1, 51, 52, 204, 205, 819, 820])  # 5,120 and 20,480 triangles
@pytest.mark.parametrize("subdiv", [4, 5])
def test_few_queries(orc, subdiv, n):
    v, idx = synth.star(subdiv, seed=6)
    q = synth.mixed_points(v, idx, n, seed=n)
    for accel, sign, am in (("rtree", "normal", A.rtree()), ("rtree_bvh", "raycast", A.rtree_bvh()),
                            ("bvh", "normal", A.bvh(S.Normal)), ("bvh", "raycast", A.bvh(S.Raycast))):
        got = m2s.generate_sdf(v, m2s.Topology.TriangleList(idx), q, am)
        assert np.array_equal(got.view(np.uint32), orc.generate_sdf(v, idx, q, accel, sign).view(np.uint32)), accel
