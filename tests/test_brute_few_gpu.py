"""None(Raycast) on small meshes, bit for bit against the oracle: the kernel for few triangles and the packed one with
short tiles, at the triangle and query counts where one gives way to the other."""
import numpy as np
import pytest

import mesh_to_sdf_b200 as m2s
from mesh_to_sdf_b200 import synth

pytestmark = pytest.mark.gpu
AM = m2s.AccelerationMethod.none(m2s.SignMethod.Raycast)


@pytest.mark.parametrize("tris,n", [(1, 1), (1, 700), (7, 513), (48, 1000), (49, 1000), (49, 49151), (49, 49152), (224, 49152),
                                    (225, 49152), (65, 1), (129, 300), (320, 5000), (1000, 513), (4, 200000), (150, 223696),
                                    (150, 223697)])
def test_small_meshes(orc, tris, n):
    v, idx = synth.star(3, seed=4)
    rng = np.random.default_rng(tris + n)
    keep = idx.reshape(-1, 3)[rng.permutation(len(idx) // 3)[:tris]]
    keep[:: 5, 1] = keep[:: 5, 0]  # some of no area
    keep = keep.reshape(-1)
    q = synth.mixed_points(v, idx, n, seed=n % 997)
    q[0] = v[keep[0]]
    far = np.array([[1e30, 0, 0], [-3e19, 1e19, 0], [1e-30, 0, 1e-38], [2e38, 2e38, 2e38]], np.float32)
    q[1:5] = far[:max(0, min(4, n - 1))]  # squares overflow; denormal
    got = m2s.generate_sdf(v, m2s.Topology.TriangleList(keep), q, AM)
    exp = orc.generate_sdf(v, keep, q, "none", "raycast")
    assert np.array_equal(got.view(np.uint32), exp.view(np.uint32))


# blocks of queries and tiles that just fill the GPU (592 blocks), fill it a little more than once and four times
@pytest.mark.parametrize("tris,n", [(4602, 4500), (4602, 4097), (8186, 3000), (19994, 1024), (19994, 7000), (1280, 60000),
                                    (300, 303105)])
def test_blocks_that_fit_at_once(orc, tris, n):
    v, idx = synth.star(5, seed=9)
    keep = idx[:3 * tris]
    q = synth.mixed_points(v, idx, n, seed=n % 997)
    got = m2s.generate_sdf(v, m2s.Topology.TriangleList(keep), q, AM)
    exp = orc.generate_sdf(v, keep, q, "none", "raycast")
    assert np.array_equal(got.view(np.uint32), exp.view(np.uint32))
