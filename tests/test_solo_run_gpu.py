"""Propagation rounds that one block relaxes alone: the same bits as with every
round on every block, for each size of the block (256, 512 and 1,024 threads by
the grid's cells) and for runs that end at different list sizes."""
import numpy as np
import pytest

import mesh_to_sdf_b200 as m2s
from mesh_to_sdf_b200 import SignMethod as S
from mesh_to_sdf_b200 import Topology as T
from mesh_to_sdf_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [S.Raycast, S.Normal])
@pytest.mark.parametrize("cells", [(40, 44, 36), (72, 70, 68), (210, 208, 200)])
def test_runs_of_one_block_give_the_same_bits(cells, sign):
    v, idx = synth.terrain(48, seed=9) if sign == S.Normal else synth.icosphere(1)
    lo, hi = synth.padded_bbox(v)
    grid = m2s.Grid.from_bounding_box(lo, hi, list(cells))
    topo = T.TriangleStrip(idx) if sign == S.Normal else T.TriangleList(idx)
    ref, alone = None, {}
    try:
        for solo in (0, 1, 7, 20, 64):
            m2s.set_grid_tuning(solo_max=solo)
            out = m2s.generate_grid_sdf(v, topo, grid, sign).view(np.uint32)
            alone[solo] = m2s.last_grid_stats()["solo_rounds"]
            ref = out if ref is None else ref
            assert np.array_equal(out, ref), solo
    finally:
        m2s.set_grid_tuning()
    assert alone[0] == 0 and alone[64] > 0, alone
