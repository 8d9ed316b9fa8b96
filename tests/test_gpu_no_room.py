"""Calls that the device has no room for (a bound on the engine's blocks stands
for a device that is nearly full): what they leave behind, and those that do
with less.
"""
import numpy as np
import pytest

import graphee_gb300 as gx
import gx_oracle as O

pytestmark = pytest.mark.gpu


def test_bounds_are_checked():
    with gx.Engine() as e:
        for which, value in ((gx.BOUND_BLOCK, -1), (99, 1)):
            with pytest.raises(gx.GxError) as ei:
                e.set_bound(which, value)
            assert ei.value.status == gx.GX_ERR_INVALID


@pytest.mark.parametrize("relabel", [0, 1])
def test_out_edges_after_a_rebuild_that_failed(relabel):
    """CC built the out-edge CSR; weighted SSSP replaces it by one with weights, and fails."""
    g = gx.rmat_graph(12, 8, seed=5, P=4, weight_seed=6)
    a = (g.V, g.P, g.bounds, g.off, g.col, g.outdeg)
    labels = O.run(O.CC, *a, 1000)[0]
    with gx.Engine(relabel=relabel, push_edge_fraction=1.0) as e:
        e.load(g)
        e.run(gx.APP_CC, 1000)
        assert np.array_equal(e.values(), labels)
        for room in (4 * g.E, 4 * g.V):
            e.set_bound(gx.BOUND_BLOCK, room)
            with pytest.raises(gx.GxError) as ei:
                e.run(gx.APP_SSSP, 1000, source=1, weighted=True)
            assert ei.value.status == gx.GX_ERR_OOM
            e.set_bound(gx.BOUND_BLOCK, 0)
            st = e.run(gx.APP_CC, 1000)
            assert np.array_equal(e.values(), labels) and st["push_iterations"] > 0
        e.run(gx.APP_SSSP, 1000, source=1, weighted=True)
        assert np.array_equal(e.values(), O.run(O.SSSP, *a, 1000, weights=g.weights, source=1)[0])


@pytest.mark.parametrize("weighted", [False, True])
def test_streaming_slots_of_one_shard(weighted):
    """No room for slots that hold a group of shards (4 M edges): they hold the longest shard, as the others did."""
    src, dst = gx.rmat_edges(16, 4 << 20, 8)
    off, col = gx.build_csc(1 << 16, src, dst)
    g = gx.Graph(1 << 16, off, col, None, 16)
    a = (g.V, g.P, g.bounds, g.off, g.col, g.outdeg)
    if weighted:
        g.weights = gx.edge_weights(3, g)
    room = 2 << 20
    assert 4 * g.E > room > 4 * np.diff(g.off[g.bounds]).max() + 64
    with gx.Engine(cache_budget_bytes=0, compress_cache=0) as e:
        e.set_bound(gx.BOUND_BLOCK, room)
        e.load(g)
        st = e.run(gx.APP_SSSP, 1000, source=1, weighted=weighted)
        assert np.array_equal(e.values(), O.run(O.SSSP, *a, 1000, weights=g.weights, source=1)[0])
        assert st["pull_launches"] >= g.P // 2  # several groups a step


@pytest.mark.parametrize("parts", [2, 7])
def test_batch_in_parts(parts):
    """No room for all instances' lists at once: part of them after part, the same results; none for one: an error."""
    g, vb = gx.batch_graph(48, scales=(6, 13), edge_factors=(8, 16), seed=5)
    with gx.Engine() as e:
        e.load(g)
        want = e.batch_run(vb, 20, 1000)
        assert want[4]["kernel_launches"] == 1
        e.set_bound(gx.BOUND_BLOCK, 64 * g.V // parts + 100000)
        got = e.batch_run(vb, 20, 1000, tuning={"threads": 256})
        assert got[4]["kernel_launches"] >= parts
        for x, y in zip(got[:4], want[:4]):
            assert np.array_equal(x, y)
        best, ms = e.batch_autotune(vb, 2, 5)
        assert ms > 0
        e.set_bound(gx.BOUND_BLOCK, 60 * 64)
        with pytest.raises(gx.GxError) as ei:
            e.batch_run(vb, 20, 1000)
        assert ei.value.status == gx.GX_ERR_OOM


def test_batch_in_parts_checks_all_first():
    """An edge that leaves the last instance: an error before the first part's results are written."""
    g, vb = gx.batch_graph(16, scales=(10, 10), edge_factors=(8, 8), seed=2)
    wrong = vb.copy()
    wrong[-2] += 100
    with gx.Engine() as e:
        e.load(g)
        for room in (0, 30 * g.V):
            e.set_bound(gx.BOUND_BLOCK, room)
            pr = np.full(g.V, 7, np.float32)
            st = gx.lib().gx_batch_run(e._h, 16, gx._ptr(wrong), 5, 5, 0.85, None, gx._ptr(pr), None, None, None, None)
            assert st == gx.GX_ERR_INVALID and (pr == 7).all()


@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("V", [1, 5, 4096, (1 << 18) + 5])
def test_triangles_packed(V, relabel):
    """No room for N+ in the CSC's spacing: counted, packed and the same triangles; unranked and ranked ids."""
    m = 12 * V if V < 1 << 18 else V // 2
    src, dst = gx.rmat_edges(max(1, int(np.ceil(np.log2(V)))), max(m, 1), V)
    hub = np.arange(V)
    src = np.concatenate([src % V, np.zeros(V, np.int64), hub])
    dst = np.concatenate([dst % V, hub, (hub + 1) % V])
    off, col = gx.build_csc(V, src, dst, gx.BUILD_DROP_SELF | gx.BUILD_DEDUP | gx.BUILD_SYMMETRIZE)
    g = gx.Graph(V, off, col, None, 3)
    with gx.Engine(relabel=relabel) as e:
        e.load(g)
        want, st = e.triangle_count()
        if V > 5:
            assert want > V // 2
            # 32 bytes a vertex (36, and the sort's 17, where ranked) and 4 an entry of N+ have room, one by one.
            e.set_bound(gx.BOUND_BLOCK, 80 * V)
            got, packed = e.triangle_count()
            assert got == want and packed["edges_scanned"] == st["edges_scanned"]
            assert packed["kernel_launches"] == st["kernel_launches"] + 3
        e.set_bound(gx.BOUND_BLOCK, 200)
        with pytest.raises(gx.GxError) as ei:
            e.triangle_count()
        assert ei.value.status == gx.GX_ERR_OOM


@pytest.mark.parametrize("weighted", [False, True])
def test_out_edges_without_room_for_buckets(weighted):
    """Room for the out-edge CSR, not for the buckets' copy of its edges: built in one pass."""
    src, dst = gx.rmat_edges(17, 6 << 20, 8)
    off, col = gx.build_csc(1 << 17, src, dst)
    g = gx.Graph(1 << 17, off, col, None, 16)
    assert g.E >= 4 << 20
    g.weights = gx.edge_weights(3, g)
    a = (g.V, g.P, g.bounds, g.off, g.col, g.outdeg)
    with gx.Engine(push_edge_fraction=1.0) as e:
        e.load(g)
        e.set_bound(gx.BOUND_BLOCK, 5 * g.E)
        st = e.run(gx.APP_SSSP, 1000, source=1, weighted=weighted)
        assert st["push_iterations"] == st["iterations"]
        ref = O.run(O.SSSP, *a, 1000, weights=g.weights if weighted else None, source=1)[0]
        assert np.array_equal(e.values(), ref)
