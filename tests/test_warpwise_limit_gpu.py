"""Point batches around the sizes where a warp per query gives way to a thread per query, bit for bit against the oracle.

The limit depends on the method and on the mesh (up to 2^15 triangles, up to 2^16, above)."""
import numpy as np
import pytest

import mesh_to_sdf_b200 as m2s
from mesh_to_sdf_b200 import synth

pytestmark = pytest.mark.gpu
A, S = m2s.AccelerationMethod, m2s.SignMethod
METHODS = {"rtree": ("rtree", "normal", A.rtree()), "rtree_bvh": ("rtree_bvh", "raycast", A.rtree_bvh()),
           "bvh_raycast": ("bvh", "raycast", A.bvh(S.Raycast)), "bvh_normal": ("bvh", "normal", A.bvh(S.Normal))}


# 31,746, 44,994 and 71,436 triangles
@pytest.mark.parametrize("edge", [126, 150, 189])
@pytest.mark.parametrize("n,methods", [(4096, ("rtree",)), (4097, ("rtree",)), (5120, ("bvh_normal",)),
                                       (5121, ("bvh_normal",)), (6144, ("rtree",)), (6145, ("rtree",)),
                                       (8192, ("rtree_bvh", "bvh_raycast", "bvh_normal")),
                                       (8193, ("rtree_bvh", "bvh_raycast", "bvh_normal")),
                                       (10240, ("rtree", "rtree_bvh")), (10241, ("rtree", "rtree_bvh"))])
def test_around_the_limits(orc, edge, n, methods):
    v, idx = synth.terrain(edge, seed=3)
    q = np.random.default_rng(n).uniform([-0.1, -0.1, -0.3], [1.1, 1.1, 0.5], (n, 3)).astype(np.float32)
    for method in methods:
        accel, sign, am = METHODS[method]
        got = m2s.generate_sdf(v, m2s.Topology.TriangleStrip(idx), q, am)
        exp = orc.generate_sdf(v, idx, q, accel, sign, strip=True)
        assert np.array_equal(got.view(np.uint32), exp.view(np.uint32)), method
