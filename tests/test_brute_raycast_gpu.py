"""None(Raycast): two queries a thread, tiles of 64 triangles, bit for bit against the oracle.

Triangle and query counts around the tile, the pair, the block (512 queries) and the Morton order (1,024 queries and
2^24 pairs)."""
import numpy as np
import pytest

import mesh_to_sdf_b200 as m2s
from mesh_to_sdf_b200 import synth

pytestmark = pytest.mark.gpu
NONE = m2s.AccelerationMethod.none(m2s.SignMethod.Raycast)


def check(orc, v, idx, q):
    got = m2s.generate_sdf(v, m2s.Topology.TriangleList(idx), q, NONE)
    exp = orc.generate_sdf(v, idx, q, "none", "raycast")
    bad = np.nonzero(got.view(np.uint32) != exp.view(np.uint32))[0]
    assert len(bad) == 0, (len(bad), q[bad[:3]], got[bad[:3]], exp[bad[:3]])


@pytest.mark.parametrize("n", [1, 2, 3, 511, 512, 513, 1025])
@pytest.mark.parametrize("tris", [1, 63, 64, 65, 129, 1280])
def test_counts(orc, tris, n):
    v, idx = synth.star(3, seed=4)
    check(orc, v, idx[:3 * tris], synth.mixed_points(v, idx, n, seed=n))


@pytest.mark.parametrize("n", [1023, 1024, 4097])
def test_morton_order(orc, n):
    v, idx = synth.star(5, seed=1)  # 20,480 triangles
    check(orc, v, idx, synth.mixed_points(v, idx, n, seed=2))


@pytest.mark.parametrize("scale,offset", [(1.0, 0.0), (1e-3, 1.0), (1.0, 1e3), (1e3, 1e5)])
def test_scales(orc, scale, offset):
    # near and far against the triangles, needles and flat ones among them
    rng = np.random.default_rng(int(offset) + 1)
    c = rng.normal(size=(700, 3))
    e = rng.normal(size=(700, 2, 3)) * rng.choice([0.02, 0.3], (700, 1, 1))
    e[::5, 1] = e[::5, 0] * 0.99 + rng.normal(size=(140, 3)) * 1e-3
    e[::31, 1] = 0
    v = (np.stack([c, c + e[:, 0], c + e[:, 1]], 1).reshape(-1, 3) * scale + offset).astype(np.float32)
    q = np.concatenate([rng.normal(size=(1500, 3)) * f for f in (0.5, 2, 30)]) * scale + offset
    check(orc, v, np.arange(len(v), dtype=np.uint32), q.astype(np.float32))
