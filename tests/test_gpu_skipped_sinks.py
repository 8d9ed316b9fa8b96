"""Standard PageRank whose selective steps skip shards: the sinks of a skipped
shard keep their rank, and the mass they hold still comes back to every vertex.
"""
import numpy as np
import pytest

import graphee_gb300 as gx

pytestmark = pytest.mark.gpu

LAYOUTS = {"resident": dict(), "relabelled": dict(relabel=1), "streamed": dict(cache_budget_bytes=0, compress_cache=0),
           "compressed": dict(cache_budget_bytes=0), "half": dict(cache_budget_bytes=16000, compress_cache=0)}


def graph():
    """Ids in quarters, four shards each: an R-MAT graph; vertices without edges; a hub's sinks and a sink with a long
    list; that list's sources."""
    n = 1024
    src, dst = gx.rmat_edges(10, 6 * n, 3)
    roots = 3 * n + np.arange(700)
    src = np.concatenate([src, roots, np.full(300, 2 * n)])
    dst = np.concatenate([dst, np.full(700, 2 * n + 900), 2 * n + 1 + np.arange(300)])
    off, col = gx.build_csc(4 * n, src, dst)
    return gx.Graph(4 * n, off, col, None, 16, np.arange(0, 4 * n + 1, n // 4))


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("heavy", [32, 4096])
def test_mass_of_skipped_sinks(layout, heavy):
    g = graph()
    sinks = g.outdeg == 0
    with gx.Engine(selective_threshold=2.0, heavy_degree=heavy, **LAYOUTS[layout]) as e:
        e.load(g)
        e.run(gx.APP_CC, 1)  # resident engines: the out-edge CSR, so that PageRank's selective steps mark shards
        skipped = 0
        for steps in range(1, 9):
            e.run(gx.APP_PAGERANK_STD, steps)
            s = e.iter_stats(steps - 1)
            skipped += s["shards_active"] < g.P
            held = float(e.values()[sinks].astype(np.float64).sum())
            # Each vertex's rank is rounded to 2^-31 / V: V of them to 2^-31.
            assert abs(s["dangling"] - held) <= 2.0**-31 + 1e-12, (steps, s)
        assert skipped >= 5
