"""Engines on several host threads at once, one to a thread: every call's results
are those it has alone.
"""
import threading

import numpy as np
import pytest

import graphee_gb300 as gx

pytestmark = pytest.mark.gpu

ROUNDS = 40


def together(*works):
    """Each work, a function of nothing, ROUNDS times on a thread of its own; what they returned or raised."""
    out = [[] for _ in works]
    start = threading.Barrier(len(works))

    def go(work, got):
        start.wait()
        for _ in range(ROUNDS):
            try:
                got.append(work())
            except gx.GxError as ex:
                got.append(ex)

    threads = [threading.Thread(target=go, args=x) for x in zip(works, out)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return out


def engine(g):
    e = gx.Engine()
    e.load(g)
    return e


def check(works, equal):
    alone = [work() for work in works]
    for got, want in zip(together(*works), alone):
        for r in got:
            assert not isinstance(r, gx.GxError) and equal(r, want), r


def test_captures_beside_frees():
    """A run's capture on one thread while the other thread's load frees memory, in turn."""
    graphs = [gx.rmat_graph(scale, 8, seed=scale, P=4) for scale in (10, 13)]
    engines = [engine(g) for g in graphs]

    def loads_and_runs(e, g):
        e.load(g)
        e.run(gx.APP_CC, 1000)
        return e.values().copy()

    check([lambda e=e, g=g: loads_and_runs(e, g) for e, g in zip(engines, graphs)], np.array_equal)
    check([lambda e=e: e.ppr(np.arange(4), 5)[0] for e in engines], np.array_equal)


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def test_batches_of_different_schedules():
    """One schedule's tables take all of an SM's shared memory, the other's a part."""
    works = []
    for n, scales, tuning in ((64, (10, 14), {"threads": 1024, "ctas_per_sm": 1}),
                              (8, (6, 8), {"threads": 256, "ctas_per_sm": 4})):
        g, vb = gx.batch_graph(n, scales=scales, edge_factors=(8, 16), seed=n)
        works.append(lambda e=engine(g), vb=vb, t=tuning: e.batch_run(vb, 20, 1000, tuning=t)[:4])
    check(works, same)


def test_triangles_of_different_sizes():
    """The larger bitmap needs more shared memory."""
    graphs = [gx.rmat_graph(scale, 8, seed=scale, P=4, symmetric=True) for scale in (12, 17)]
    check([lambda e=engine(g): e.triangle_count()[0] for g in graphs], int.__eq__)


def test_out_edges_of_different_sizes():
    """A load's first CC run builds the out-edge CSR: 8 buckets of sources for one graph, 320 for the other."""
    works = []
    for V in (1 << 17, 40 << 17):
        off, col = gx.build_csc(V, *gx.rmat_edges(17, 6 << 20, V))
        g = gx.Graph(V, off, col, None, 4)
        assert g.E >= 4 << 20

        def work(e=engine(g), g=g):
            e.load(g)
            e.run(gx.APP_CC, 1000)
            return e.values().copy()

        works.append(work)
    check(works, np.array_equal)


def test_hot_tables_of_different_sizes():
    g = gx.rmat_graph(16, 8, seed=3, P=4)
    works = []
    for hot in (64, 40000):
        e = gx.Engine(hot_vertices=hot)
        e.load(g)
        works.append(lambda e=e: (e.run(gx.APP_PAGERANK_REF, 8), e.values().copy())[1])
    check(works, np.array_equal)
