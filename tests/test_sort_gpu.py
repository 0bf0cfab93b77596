"""The radix sort at the edges of its tiles and passes, bit for bit against a stable sort."""
import numpy as np
import pytest

import mesh_to_sdf_b200 as m2s

pytestmark = pytest.mark.gpu


def keys_of(kind, n, bits, rng):
    top = (1 << bits) - 1
    if kind == "random":
        return rng.integers(0, top + 1, n, dtype=np.uint64).astype(np.uint32)
    if kind == "equal":
        return np.full(n, top & 0xA5A5A5A5, np.uint32)
    if kind == "falling":
        return (top - np.minimum(np.arange(n, dtype=np.uint64), top)).astype(np.uint32)
    return (rng.integers(0, 3, n) * (top // 2)).astype(np.uint32)  # few values


# 2,048 and 8,192: the tiles; 2^20: from there the large ones
@pytest.mark.parametrize("n", [2, 31, 2047, 2048, 2049, 8193, 100003, (1 << 20) - 1, 1 << 20, (1 << 20) + 8191, 3000001])
@pytest.mark.parametrize("kind,bits", [("random", 32), ("random", 30), ("random", 7), ("random", 17), ("equal", 32),
                                       ("falling", 32), ("few", 24)])
def test_pairs(n, kind, bits):
    import torch

    rng = np.random.default_rng(n + bits)
    keys = keys_of(kind, n, bits, rng)
    vals = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    k, v = (torch.from_numpy(x.view(np.int32).copy()).cuda() for x in (keys, vals))
    m2s.radix_sort_pairs_device(k, v, bits)
    torch.cuda.synchronize()
    # only whole digits are looked at: the keys lie below 2^bits
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k.cpu().numpy().view(np.uint32), keys[order])
    assert np.array_equal(v.cpu().numpy().view(np.uint32), vals[order])


@pytest.mark.parametrize("n", [1, 2, 2049, 1 << 20, 1500001])
def test_floats(n):
    rng = np.random.default_rng(n)
    d = rng.normal(size=n).astype(np.float32)
    d[rng.integers(0, n, n // 3)] = np.float32(-0.0)
    d[rng.integers(0, n, n // 5)] = np.float32(0.5)
    if n > 100:
        d[rng.integers(0, n, 9)] = [np.nan, -np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-40, -1e-40, 3e38]
    order, (lo, hi) = m2s.sort_cells_by_distance(d)
    b = d.view(np.uint32)
    key = np.where(b >> 31, ~b, b | np.uint32(0x80000000))
    assert np.array_equal(order, np.argsort(key, kind="stable").astype(np.uint32))
    ok = d[~np.isnan(d)]
    assert lo == ok.min() and hi == ok.max()
