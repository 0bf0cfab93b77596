"""m2s_generate_sdf_none_noalloc, Raycast, where several blocks share a query's triangles and merge in the output: bit for
bit what the allocating entry point gives.  Sizes at the edges of a tile (64 triangles), of a block (512 queries) and
of the number of chunks (2,368 blocks, 256 chunks)."""
import ctypes

import numpy as np
import pytest

import mesh_to_sdf_b200 as m2s
from mesh_to_sdf_b200 import _lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tris", [1, 63, 64, 65, 129, 1280, 20480])
@pytest.mark.parametrize("n", [1, 2, 511, 512, 513, 5000])
def test_merged_chunks(tris, n):
    import torch

    v, idx = synth.star(5 if tris > 1280 else 3, seed=7)
    keep = idx.reshape(-1, 3)[:tris].reshape(-1)
    lo, hi = synth.padded_bbox(v)
    q = synth.uniform_points(n, lo, hi, seed=n)
    q[0] = 1e30  # far: its squared distances overflow and stay at f32::MAX
    exp = m2s.generate_sdf(v, m2s.Topology.TriangleList(keep), q, m2s.AccelerationMethod.none(m2s.SignMethod.Raycast))
    vd, qd = torch.from_numpy(v).cuda(), torch.from_numpy(q).cuda()
    kd = torch.from_numpy(keep.astype(np.int32)).cuda()
    for _ in range(2):
        out = torch.full((n,), float("nan"), device="cuda")
        st = _lib.lib().m2s_generate_sdf_none_noalloc(
            ctypes.c_void_p(vd.data_ptr()), len(v), ctypes.c_void_p(kd.data_ptr()), len(keep), 32, 0,
            ctypes.c_void_p(qd.data_ptr()), n, 0, ctypes.c_void_p(out.data_ptr()), None)
        assert st == 0
        assert np.array_equal(out.cpu().numpy().view(np.uint32), exp.view(np.uint32))
