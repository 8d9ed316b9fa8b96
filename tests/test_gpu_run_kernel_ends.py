"""How PageRank's one-launch supersteps end: their barrier gives up after its
polls and the engine runs again; they hand over to selective steps where the
step-by-step launches turn selective, with the same edges read and shards swept;
and they are what runs.
"""
import numpy as np
import pytest

import graphee_gb300 as gx
import gx_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("app", [gx.APP_PAGERANK_REF, gx.APP_PAGERANK_STD])
def test_barrier_timeout_then_recovery(app):
    g = gx.rmat_graph(17, 16, seed=4, P=8)
    with gx.Engine() as e:
        e.load(g)
        e.run(app, 20)
        want = e.values().copy()
        e.set_bound(gx.BOUND_RUN_POLLS, 1)
        with pytest.raises(gx.GxError) as ei:
            e.run(app, 20)
        assert ei.value.status == gx.GX_ERR_TIMEOUT
        e.set_wait_limit(1)  # bounds other calls' waits, not this one's
        e.set_bound(gx.BOUND_RUN_POLLS, 0)
        e.run(app, 20)
        assert np.array_equal(e.values().view(np.uint32), want.view(np.uint32))
        e.run(gx.APP_CC, 1000)
        assert np.array_equal(e.values(), O.run(O.CC, g.V, g.P, g.bounds, g.off, g.col, g.outdeg, 1000)[0])


def test_polls_are_checked():
    with gx.Engine() as e:
        with pytest.raises(gx.GxError) as ei:
            e.set_bound(gx.BOUND_RUN_POLLS, 1 << 32)
        assert ei.value.status == gx.GX_ERR_INVALID


@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("V,P", [(1000, 4), (20011, 37), (200003, 64)])
def test_same_edges_and_shards(V, P, relabel):
    src, dst = gx.rmat_edges(int(np.ceil(np.log2(V))), 8 * V, V)
    keep = (src < V) & (dst < V)
    off, col = gx.build_csc(V, src[keep], dst[keep])
    g = gx.Graph(V, off, col, None, P)
    # Ends in dense steps, in selective ones soon and late, in the first batch of eight and at its ends.
    runs = [(gx.APP_PAGERANK_REF, 0.001, dict(max_iter=20)), (gx.APP_PAGERANK_STD, 0.001, dict(max_iter=70)),
            (gx.APP_PAGERANK_REF, 0.001, dict(max_iter=200)), (gx.APP_PAGERANK_STD, 0.5, dict(max_iter=200)),
            (gx.APP_PAGERANK_REF, 0.9, dict(max_iter=24)), (gx.APP_PAGERANK_REF, 2.0, dict(max_iter=9)),
            (gx.APP_PAGERANK_STD, 0.001, dict(max_iter=150, tolerance=1e-5))]
    for app, threshold, prm in runs:
        got = []
        for use_graph in (1, 0):
            with gx.Engine(relabel=relabel, use_graph=use_graph, selective_threshold=threshold) as e:
                e.load(g)
                st = e.run(app, **prm)
                steps = [e.iter_stats(i) for i in range(st["iterations"])]
                got.append((st["iterations"], st["edges_scanned"], steps, e.values().view(np.uint32).copy()))
                if use_graph and all(s["mode"] == 0 for s in steps):  # init_kernel, and 64 steps to a launch
                    assert st["kernel_launches"] == 1 + (st["iterations"] + 63) // 64
                if not use_graph:
                    assert st["kernel_launches"] >= 2 * st["iterations"]
        assert got[0][:3] == got[1][:3], (app, threshold, prm)
        assert np.array_equal(got[0][3], got[1][3]), (app, threshold, prm)
