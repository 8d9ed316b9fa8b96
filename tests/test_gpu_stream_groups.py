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
