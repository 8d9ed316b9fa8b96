"""Work-unit sizes and launch shapes of the pull kernel at their edges: graphs
with fewer units than warps (a unit per warp), about as many, and more (claimed
units), in-lists around every cap, in both layouts, against the oracle.
"""
import numpy as np
import pytest

import graphee_gb300 as gx
import gx_oracle as O

pytestmark = pytest.mark.gpu

# 152 SMs x 32 warps, a tile of up to 32 vertices each.
WARPS = 4864


def graph(V, lists, P, fill):
    """`fill` in-edges for every vertex, and the given in-list lengths from vertex 0 on."""
    rng = np.random.default_rng(V + len(lists))
    n = np.minimum(np.full(V, fill), V)
    n[:len(lists)] = np.minimum(lists, V)
    dst = np.repeat(np.arange(V, dtype=np.int32), n)
    src = np.concatenate([rng.permutation(V)[:k] if k > fill else rng.integers(0, V, k) for k in n[:len(lists)]] +
                         [rng.integers(0, V, int(n[len(lists):].sum()))]).astype(np.int32)
    off, col = gx.build_csc(V, src, dst)
    g = gx.Graph(V, off, col, None, P)
    g.weights = gx.edge_weights(3, g)
    return g


EDGES = [15, 16, 17, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1025, 2047, 2049, 4097, 8192]


@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("V,lists,fill", [(1, [], 0), (31, [], 3), (33, [33], 5), (10007, EDGES, 2),
                                          (32 * WARPS - 32, EDGES, 1), (32 * WARPS + 33, EDGES, 1),
                                          (3 * 32 * WARPS + 1, EDGES[::-1], 2)])
def test_units(V, lists, fill, relabel):
    g = graph(V, lists, min(7, V), fill)
    a = (g.V, g.P, g.bounds, g.off, g.col, g.outdeg)
    ref, _, _ = O.run(O.PAGERANK_REF, *a, 12)
    dst = np.repeat(np.arange(V), np.diff(g.off))
    exact = np.full(V, 1.0 / V)
    for _ in range(12):
        exact = 0.85 * np.bincount(dst, (exact / np.maximum(g.outdeg, 1))[g.col], V) + 1.0 / V
    with gx.Engine(relabel=relabel) as e:
        e.load(g)
        e.run(gx.APP_PAGERANK_REF, 12)
        ranks = e.values().astype(np.float64)
        # The parity bound, against 64-bit sums: on lists of thousands of edges
        # the reference's own sequential FP32 sum is further off than that.
        assert np.max(np.abs(ranks - exact) / exact) < 1e-5
        e.run(gx.APP_CC, 1000)
        assert np.array_equal(e.values(), O.run(O.CC, *a, 1000)[0])
        e.run(gx.APP_SSSP, 1000, source=V // 2, weighted=True)
        assert np.array_equal(e.values(), O.run(O.SSSP, *a, 1000, weights=g.weights, source=V // 2)[0])
    with gx.Engine(relabel=relabel, exact_order=1) as e:
        e.load(g)
        e.run(gx.APP_PAGERANK_REF, 12)
        assert np.array_equal(e.values().view(np.uint32), ref.view(np.uint32))


# Out-degrees around a frontier entry (256 edges), around what a lane of the
# compaction writes itself (8 entries) and beyond a warp's 32 entries.
HUBS = [1, 255, 256, 257, 2047, 2048, 2049, 2305, 8192, 8193, 40000]


@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("copies", [1, 40, 600])
def test_push_hubs(copies, relabel):
    """The source reaches `copies` of each hub in step 0, which reach the rest in step 1."""
    V = 60000
    rng = np.random.default_rng(copies)
    lists = np.array(HUBS * copies)[:1 + 2_000_000 // 5000]
    hub = 1 + np.arange(len(lists))
    src = np.concatenate([np.zeros(len(lists), np.int64), np.repeat(hub, lists)])
    dst = np.concatenate([hub] + [rng.permutation(V)[:n] for n in lists])
    off, col = gx.build_csc(V, src, dst)
    g = gx.Graph(V, off, col, None, 5)
    g.weights = gx.edge_weights(9, g)
    a = (g.V, g.P, g.bounds, g.off, g.col, g.outdeg)
    with gx.Engine(relabel=relabel, push_edge_fraction=1.0) as e:
        e.load(g)
        for weighted in (True, False):
            st = e.run(gx.APP_SSSP, 1000, source=0, weighted=weighted)
            ref, changed, _ = O.run(O.SSSP, *a, 1000, weights=g.weights if weighted else None, source=0)
            assert np.array_equal(e.values(), ref)
            assert [e.iter_stats(i)["changed"] for i in range(st["iterations"])] == list(changed)
            assert st["push_iterations"] == st["iterations"]


@pytest.mark.parametrize("relabel", [0, 1])
def test_out_edges_by_buckets(relabel):
    """Enough edges for the bucketed transpose: buckets of one slice and of several, hubs among sources and
    destinations, a last bucket that is not full.  Weighted distances and labels depend on every out-edge."""
    V, n = 5 * 16384 + 77, 5 << 20
    rng = np.random.default_rng(4)
    src = np.concatenate([rng.integers(0, V, n), np.repeat([0, 16383, 16384, V - 1], V), rng.integers(0, 16384, n // 4)])
    dst = np.concatenate([rng.integers(0, V, n), np.tile(np.arange(V), 4), np.minimum(rng.integers(0, V, n // 4), 99)])
    off, col = gx.build_csc(V, src, dst)
    g = gx.Graph(V, off, col, None, 9)
    g.weights = gx.edge_weights(2, g)
    assert g.E > 4 << 20
    a = (g.V, g.P, g.bounds, g.off, g.col, g.outdeg)
    with gx.Engine(relabel=relabel, push_edge_fraction=1.0) as e:
        e.load(g)
        for source in (1, V - 2):
            st = e.run(gx.APP_SSSP, 1000, source=source, weighted=True)
            assert st["push_iterations"] == st["iterations"]
            assert np.array_equal(e.values(), O.run(O.SSSP, *a, 1000, weights=g.weights, source=source)[0])
        e.run(gx.APP_CC, 1000)
        assert np.array_equal(e.values(), O.run(O.CC, *a, 1000)[0])
