"""PageRank's one-launch supersteps against the step-by-step launches: the
same ranks bit for bit, the same steps and per-step counts, for runs that end
by their step limit, by the tolerance, by convergence or in selective steps,
in one launch or several, resumed or not, in both layouts.
"""
import numpy as np
import pytest

import graphee_gb300 as gx

pytestmark = pytest.mark.gpu


def graph(V, P):
    if V < 100:
        src, dst = np.arange(V), (np.arange(V) * 3 + 1) % V
    else:
        src, dst = gx.rmat_edges(int(np.ceil(np.log2(V))), 12 * V, V)
        src, dst = src[(src < V) & (dst < V)], dst[(src < V) & (dst < V)]
    off, col = gx.build_csc(V, src, dst)
    return gx.Graph(V, off, col, None, P)


@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("V,P", [(1, 1), (33, 2), (1000, 4), (20011, 3), (200003, 64), (700001, 7)])
def test_same_as_step_by_step(V, P, relabel):
    g = graph(V, P)
    start = np.random.default_rng(V).random(V, np.float32) / np.float32(V)
    runs = [(gx.APP_PAGERANK_REF, dict(max_iter=1)), (gx.APP_PAGERANK_REF, dict(max_iter=20)),
            (gx.APP_PAGERANK_REF, dict(max_iter=150)), (gx.APP_PAGERANK_STD, dict(max_iter=64)),
            (gx.APP_PAGERANK_STD, dict(max_iter=200, tolerance=1e-4)),
            (gx.APP_PAGERANK_STD, dict(max_iter=90, use_init=True, first_step=3, damping=0.99)),
            (gx.APP_PAGERANK_REF, dict(max_iter=30, use_init=True))]
    for app, prm in runs:
        got = []
        for use_graph in (1, 0):
            with gx.Engine(relabel=relabel, use_graph=use_graph) as e:
                e.load(g)
                e.set_init(start)
                st = e.run(app, **prm)
                steps = [e.iter_stats(i) for i in range(st["iterations"])]
                got.append((st["iterations"], st["changed_last"], st["residual_l1_last"],
                            [(s["changed"], s["active"], s["mode"], s["residual_l1"], s["dangling"]) for s in steps],
                            e.values().copy()))
        a, b = got
        assert a[:4] == b[:4], (app, prm)
        assert np.array_equal(a[4].view(np.uint32), b[4].view(np.uint32)), (app, prm)
