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
