"""The radix sort's rare paths, bit for bit against a stable sort: tiles that give up looking back and count the digits
before them from the keys, and the 64-bit tile words of 2^30 pairs and more, both asked for at small sizes."""
import ctypes

import numpy as np
import pytest

from mesh_to_sdf_b200 import _lib

pytestmark = pytest.mark.gpu


# 2,048 pairs a tile below 2^20 pairs, 8,192 with 64-bit words
@pytest.mark.parametrize("n", [2, 2049, 8193, 40000, 70001])
@pytest.mark.parametrize("polls", [0, 1, 1 << 16])
@pytest.mark.parametrize("wide", [0, 1])
@pytest.mark.parametrize("bits", [30, 9])
def test_paths(n, polls, wide, bits):
    import torch

    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    keys[n // 3: n // 2] = keys[0]
    vals = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    k, v = (torch.from_numpy(x.view(np.int32).copy()).cuda() for x in (keys, vals))
    st = _lib.lib().m2s_test_radix_sort(ctypes.c_void_p(k.data_ptr()), ctypes.c_void_p(v.data_ptr()), n, bits, polls, wide,
                                        None)
    assert st == 0
    torch.cuda.synchronize()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k.cpu().numpy().view(np.uint32), keys[order])
    assert np.array_equal(v.cpu().numpy().view(np.uint32), vals[order])
