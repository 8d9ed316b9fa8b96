"""Streamed shards that travel and are swept in groups: what a run does and
reports is that of its shards one by one, and of the resident engine.
"""
import numpy as np
import pytest

import graphee_gb300 as gx

pytestmark = pytest.mark.gpu


def test_streamed_shards_counted():
    """Shards without vertices are neither copied nor counted, also inside a group; those without edges are."""
    g = gx.rmat_graph(12, 8, seed=2, P=1)
    bounds = np.array([0, 0, 500, 500, 500, 1500, 3000, 3000, 4096, 4096], np.int32)
    g = gx.Graph(g.V, g.off, g.col, g.outdeg, 9, bounds)
    with gx.Engine(cache_budget_bytes=0, compress_cache=0) as e:
        e.load(g)
        st = e.run(gx.APP_PAGERANK_REF, 3)
    assert st["shards_streamed"] == 4 * 3


def graph(P):
    """A shard in five without vertices, one without edges, the others of uneven lengths."""
    g = gx.rmat_graph(13, 12, seed=7, P=1)
    rng = np.random.default_rng(P)
    cuts = np.sort(rng.integers(0, g.V, P - 1))
    cuts[::5] = cuts[np.minimum(np.arange(P - 1)[::5] + 1, P - 2)]
    bounds = np.concatenate([[0], np.sort(cuts), [g.V]]).astype(np.int32)
    g = gx.Graph(g.V, g.off, g.col, g.outdeg, P, bounds)
    g.weights = gx.edge_weights(6, g)
    return g


RUNS = [(gx.APP_PAGERANK_REF, dict(max_iter=12)), (gx.APP_PAGERANK_STD, dict(max_iter=12)),
        (gx.APP_SSSP, dict(max_iter=1000, source=1, weighted=True)), (gx.APP_SSSP, dict(max_iter=1000, source=1)),
        (gx.APP_CC, dict(max_iter=1000))]


@pytest.mark.parametrize("threshold", [0.001, 2.0])
@pytest.mark.parametrize("exact", [0, 1])
@pytest.mark.parametrize("compress", [0, 1])
@pytest.mark.parametrize("budget", [0, 150_000, 400_000])
@pytest.mark.parametrize("group", [1, 3000, 20_000])
def test_several_groups_a_step(group, budget, compress, exact, threshold):
    """Groups cut at a few thousand edges, so that a step has many and takes every slot again: values and counts of the
    resident engine, with some shards resident, compressed or skipped."""
    g = graph(41)
    with gx.Engine(push_sparse=0, exact_order=exact, selective_threshold=threshold) as r, \
            gx.Engine(cache_budget_bytes=budget, compress_cache=compress, stream_slots=2, exact_order=exact,
                      selective_threshold=threshold) as e:
        r.load(g)
        e.set_bound(gx.BOUND_STREAM_GROUP, group)
        e.load(g)
        for app, prm in RUNS:
            a, b = r.run(app, **prm), e.run(app, **prm)
            assert a["iterations"] == b["iterations"]
            x, y = r.values().view(np.uint32), e.values().view(np.uint32)
            if app == gx.APP_PAGERANK_STD and threshold > 1:
                # The resident engine marks shards from its second batch of steps on, the streamed one at once.
                assert np.allclose(x.view(np.float32), y.view(np.float32), rtol=1e-3)
            else:
                assert np.array_equal(x, y)
                for i in range(a["iterations"]):
                    assert r.iter_stats(i)["changed"] == e.iter_stats(i)["changed"]
            most = max(group, int(np.diff(g.off[g.bounds]).max()))
            streamed = 0 if budget else g.E // (most + 8)
            assert b["pull_launches"] >= max(2, streamed if threshold < 1 else 0)
