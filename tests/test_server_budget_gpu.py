"""The server's budget and the pillboxes: they take only what the budget has to spare.

A resident mesh reserves 160 bytes a triangle, an upload 320, a point request 64 bytes a query, each request 1 MiB more;
the pillboxes' 64 bytes a triangle come on top where they fit.  So requests that the reservations leave room for are
accepted and finish, none is answered by an eviction, and the results do not depend on which meshes still hold theirs."""
import numpy as np
import pytest

import mesh_to_sdf_b200 as m2s
from mesh_to_sdf_b200 import synth

pytestmark = pytest.mark.gpu
A, S, T = m2s.AccelerationMethod, m2s.SignMethod, m2s.Topology
MB = 1 << 20


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def upload_need(v, idx):
    return 320 * (len(idx) // 3) + 12 * len(v) + 4 * len(idx) + MB


def test_request_beside_one_mesh():
    v, idx = synth.star(3, seed=2)
    lo, hi = synth.padded_bbox(v)
    q = synth.uniform_points(6000, lo, hi, seed=3)
    budget = 160 * (len(idx) // 3) + 64 * len(q) + MB  # not a byte for pillboxes
    assert budget >= upload_need(v, idx)
    srv = m2s.Server(budget)
    try:
        mid, t = srv.submit_upload(v, T.TriangleList(idx), A.rtree_bvh())
        assert srv.wait(t, timeout_s=60)[0] == 0
        out = np.empty(len(q), np.float32)
        assert srv.wait(srv.submit_points(mid, q, out), timeout_s=60)[0] == 0
        ref = m2s.query_sdf(m2s.build_sdf_acceleration(v, T.TriangleList(idx), A.rtree_bvh()), q)
        assert np.array_equal(bits(out), bits(ref))
        assert srv.stats()["reserved_bytes"] <= budget  # (its peak counts an upload and its mesh together for a moment)
    finally:
        srv.close()


# room for no pillboxes beside the third upload, for some of them, for all
@pytest.mark.parametrize("extra", [0, 400_000, 64 * MB])
def test_several_meshes(extra):
    items = [synth.star(4, seed=s) for s in (4, 5, 6)]
    methods = [A.rtree_bvh(), A.rtree(), A.bvh(S.Normal)]
    tris = len(items[0][1]) // 3
    budget = 2 * 160 * tris + max(upload_need(v, i) for v, i in items) + extra
    srv = m2s.Server(budget)
    try:
        ids = []
        for (v, idx), am in zip(items, methods):
            mid, t = srv.submit_upload(v, T.TriangleList(idx), am)
            assert srv.wait(t, timeout_s=60)[0] == 0
            ids.append(mid)
        assert srv.stats()["evictions"] == 0 and srv.stats()["resident_meshes"] == 3
        jobs = []
        for k in range(18):  # all at once: requests wait for room, and for pillboxes that running ones read
            j = k % 3
            v, idx = items[j]
            lo, hi = synth.padded_bbox(v)
            if k % 5 == 4:
                grid = m2s.Grid.from_bounding_box(lo, hi, [10, 11, 12])
                out = np.empty(grid.get_total_cell_count(), np.float32)
                jobs.append((j, grid, out, srv.submit_grid(ids[j], grid, S.Raycast, out)))
            else:
                q = synth.uniform_points(500 + 700 * k, lo, hi, seed=k)
                out = np.empty(len(q), np.float32)
                jobs.append((j, q, out, srv.submit_points(ids[j], q, out)))
        direct = [m2s.build_sdf_acceleration(v, T.TriangleList(i), am) for (v, i), am in zip(items, methods)]
        for j, arg, out, t in jobs:
            assert srv.wait(t, timeout_s=60)[0] == 0
            if isinstance(arg, m2s.Grid):
                ref = m2s.generate_grid_sdf(items[j][0], T.TriangleList(items[j][1]), arg, S.Raycast)
            else:
                ref = m2s.query_sdf(direct[j], arg)
            assert np.array_equal(bits(out), bits(ref))
        st = srv.stats()
        assert st["failed"] == 0 and st["evictions"] == 0 and st["queued"] == 0
        held = 3 * 160 * tris  # and each mesh's 64 bytes a node, as far as they fit
        assert held <= st["reserved_bytes"] <= held + 3 * 64 * (tris - 1)
        if extra >= 64 * MB:
            assert st["reserved_bytes"] == held + 3 * 64 * (tris - 1)
    finally:
        srv.close()


def test_upload_beside_a_busy_mesh():
    """An upload that only the pillboxes of a mesh with a stream of requests are in the way of."""
    (v, idx), (v2, idx2) = synth.star(4, seed=7), synth.star(4, seed=8)
    lo, hi = synth.padded_bbox(v)
    q = synth.uniform_points(60000, lo, hi, seed=3)
    tris, point = len(idx) // 3, 64 * len(q) + MB
    budget = 160 * tris + 2 * point + upload_need(v2, idx2) + 100_000  # less than the pillboxes' 327,616
    srv = m2s.Server(budget)
    try:
        mid, t = srv.submit_upload(v, T.TriangleList(idx), A.rtree_bvh())
        assert srv.wait(t, timeout_s=60)[0] == 0
        outs = [np.empty(len(q), np.float32) for _ in range(40)]
        jobs = [srv.submit_points(mid, q, o) for o in outs[:20]]
        mid2, t2 = srv.submit_upload(v2, T.TriangleList(idx2), A.rtree_bvh())
        jobs += [srv.submit_points(mid, q, o) for o in outs[20:]]
        assert srv.wait(t2, timeout_s=60)[0] == 0
        last = np.empty(1000, np.float32)
        jobs.append(srv.submit_points(mid2, q[:1000], last))
        for t in jobs:
            assert srv.wait(t, timeout_s=60)[0] == 0
        ref = m2s.query_sdf(m2s.build_sdf_acceleration(v, T.TriangleList(idx), A.rtree_bvh()), q)
        for o in outs:
            assert np.array_equal(bits(o), bits(ref))
        ref2 = m2s.query_sdf(m2s.build_sdf_acceleration(v2, T.TriangleList(idx2), A.rtree_bvh()), q[:1000])
        assert np.array_equal(bits(last), bits(ref2))
        st = srv.stats()
        assert st["failed"] == 0 and st["evictions"] == 0 and st["queued"] == 0 and st["reserved_bytes"] <= budget
    finally:
        srv.close()
