"""More pieces of large triangles than the list for them holds (it lies in the job's bucket lists: 19 x (cells + 1,024)
entries for a small grid): the triangles that do not fit stay with their own warps.

Every triangle's box covers the whole grid, so every cell sees every triangle: with Raycast the distance is the exact
nearest one, bit for bit, and the signs are the oracle's."""
import numpy as np
import pytest

import mesh_to_sdf_b200 as m2s

pytestmark = pytest.mark.gpu


def soup(n, seed):
    """Triangles whose boxes hold [-1.5, 1.5]^3."""
    rng = np.random.default_rng(seed)
    t = np.stack([rng.uniform(-3, -1.5, (n, 3)), rng.uniform(1.5, 3, (n, 3)), rng.uniform(-3, 3, (n, 3))], 1)
    return t.astype(np.float32).reshape(-1, 3), np.arange(3 * n, dtype=np.uint32)


def check(orc, sdf, v, idx, grid, sign):
    cells = grid.cell_centers()
    exact = np.abs(orc.generate_sdf(v, idx, cells, "none", "raycast"))
    if sign == "raycast":
        assert np.array_equal(np.abs(sdf).view(np.uint32), exact.view(np.uint32))
        ref = orc.generate_grid_sdf(v, idx, grid.first_cell, grid.cell_size, grid.cell_count, sign, n_threads=1)
        assert np.array_equal(np.signbit(sdf), np.signbit(ref))
    else:  # compare_distances' band is 1e-6 (or 2 ulps) wide, and a fold drifts by no more than one band
        assert (np.abs(np.abs(sdf).astype(np.float64) - exact) <= 4e-6).all()


# pieces per triangle: 3 of the box (and of the x rectangle in the second grid); the list holds 40,356 and 39,520
@pytest.mark.parametrize("count", [(11, 10, 10), (1, 33, 32)])
@pytest.mark.parametrize("tris", [13000, 14000, 20000])  # 39,000, 42,000, 60,000 pieces
def test_single(orc, count, tris):
    v, idx = soup(tris, tris)
    grid = m2s.Grid.from_bounding_box([-1] * 3, [1] * 3, count)
    for sign in ("raycast", "normal"):
        sdf = m2s.generate_grid_sdf(v, m2s.Topology.TriangleList(idx), grid, m2s.SignMethod[sign.capitalize()])
        check(orc, sdf.reshape(-1), v, idx, grid, sign)


def test_batch(orc):
    import torch

    grids = [m2s.Grid.from_bounding_box([-1] * 3, [1] * 3, c) for c in ((1, 33, 32), (11, 10, 10), (5, 5, 5))]
    soups = [soup(n, n) for n in (20000, 15000, 300)]  # 105,000 pieces, the list holds 61,959
    meshes = [m2s.build_sdf_acceleration(v, m2s.Topology.TriangleList(i)) for v, i in soups]
    off = m2s.grid_offsets(grids)
    for sign in ("raycast", "normal"):
        out = torch.full((int(off[-1]),), float("nan"), device="cuda")
        m2s.grid_sdf_batch_device(meshes, grids, m2s.SignMethod[sign.capitalize()], out)
        torch.cuda.synchronize()
        for k, (v, i) in enumerate(soups):
            check(orc, out[int(off[k]):int(off[k + 1])].cpu().numpy(), v, i, grids[k], sign)
