"""Triangles whose boxes hold many grid cells: seeding and rays split them over several warps.

The bars are those of the grid parity tests: Raycast signs cell for cell as the oracle's single-heap run, every
distance a real triangle's (not below the exact nearest one, at most a cell diagonal further above it than the
oracle's own)."""
import numpy as np
import pytest

import mesh_to_sdf_b200 as m2s
from mesh_to_sdf_b200 import synth

pytestmark = pytest.mark.gpu


def box_mesh():
    v = np.array([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)], np.float32)
    f = [(0, 1, 3), (0, 3, 2), (4, 6, 7), (4, 7, 5), (0, 4, 5), (0, 5, 1), (2, 3, 7), (2, 7, 6), (0, 2, 6), (0, 6, 4),
         (1, 5, 7), (1, 7, 3)]
    # turned, so that the faces' boxes are solid and no ray runs in a face
    rot = synth.random_rotation(np.random.default_rng(5))
    return (v.astype(np.float64) @ rot.T).astype(np.float32), np.array(f, np.uint32).reshape(-1)


# edges around the split (1,024 cells of a box or rectangle) and the chunk (512)
@pytest.mark.parametrize("count", [(10, 10, 10), (23, 24, 25), (45, 46, 47), (80, 81, 79), (1, 90, 70), (64, 3, 100)])
@pytest.mark.parametrize("mesh", ["box", "icosphere_s0", "terrain_strip"])
def test_large_triangles(orc, mesh, count):
    strip = mesh == "terrain_strip"
    v, idx = box_mesh() if mesh == "box" else synth.icosphere(0) if mesh == "icosphere_s0" else synth.terrain(6, seed=1)
    lo, hi = synth.padded_bbox(v)
    grid = m2s.Grid.from_bounding_box(lo, hi, count)
    topo = m2s.Topology.TriangleStrip(idx) if strip else m2s.Topology.TriangleList(idx)
    diag = float(np.linalg.norm(grid.cell_size.astype(np.float64)))
    exact = orc.generate_sdf(v, idx, grid.cell_centers(), "bvh", "raycast", strip=strip)
    for sign in ("raycast", "normal"):
        sdf = m2s.generate_grid_sdf(v, topo, grid, m2s.SignMethod[sign.capitalize()])
        ref = orc.generate_grid_sdf(v, idx, grid.first_cell, grid.cell_size, grid.cell_count, sign, n_threads=1,
                                    strip=strip)
        if sign == "raycast":
            assert np.array_equal(np.signbit(sdf), np.signbit(ref))
        gap = np.abs(sdf).astype(np.float64) - np.abs(exact).astype(np.float64)
        most = float((np.abs(ref).astype(np.float64) - np.abs(exact).astype(np.float64)).max()) + diag
        tol = 1e-6 * float(np.linalg.norm((hi - lo).astype(np.float64)))
        assert gap.min() >= -tol and gap.max() <= most + tol
        again = m2s.generate_grid_sdf(v, topo, grid, m2s.SignMethod[sign.capitalize()])
        assert np.array_equal(np.abs(sdf).view(np.uint32), np.abs(again).view(np.uint32))
