"""More changed hubs in a step than the launch that writes their frontier
entries has warps, each of more entries than a lane of the compaction writes.
"""
import numpy as np
import pytest

import graphee_gb300 as gx
import gx_oracle as O

pytestmark = pytest.mark.gpu

WARPS = 4864      # 152 SMs x 32
OWN = 8 * 256     # out-edges of the entries a lane writes itself


@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("hubs", [WARPS - 1, WARPS + 1, 2 * WARPS + 100])
def test_every_hub_is_expanded(hubs, relabel):
    """The source reaches the hubs in step 0; they reach the rest, each vertex first by some hub alone."""
    rng = np.random.default_rng(hubs)
    rest = 4096
    V = 1 + hubs + rest
    lists = OWN + rng.choice([0, 1, 2, 255, 256, 257], hubs)
    hub = 1 + np.arange(hubs)
    # A hub's list: consecutive vertices of the rest from a start of its own.
    at = np.repeat(rng.integers(0, rest, hubs), lists) + np.arange(lists.sum()) - np.repeat(np.cumsum(lists) - lists, lists)
    src = np.concatenate([np.zeros(hubs, np.int64), np.repeat(hub, lists)])
    dst = np.concatenate([hub, 1 + hubs + at % rest])
    off, col = gx.build_csc(V, src, dst)
    g = gx.Graph(V, off, col, None, 5)
    g.weights = gx.edge_weights(9, g)
    a = (g.V, g.P, g.bounds, g.off, g.col, g.outdeg)
    assert np.count_nonzero(g.outdeg > OWN) > hubs // 2 and np.count_nonzero(g.outdeg == OWN) > 0
    if hubs > 2 * WARPS:
        assert np.count_nonzero(g.outdeg > OWN) > WARPS
    with gx.Engine(relabel=relabel, push_edge_fraction=1.0) as e:
        e.load(g)
        for weighted in (True, False):
            st = e.run(gx.APP_SSSP, 1000, source=0, weighted=weighted)
            ref, changed, _ = O.run(O.SSSP, *a, 1000, weights=g.weights if weighted else None, source=0)
            assert np.array_equal(e.values(), ref)
            assert [e.iter_stats(i)["changed"] for i in range(st["iterations"])] == list(changed)
            assert st["push_iterations"] == st["iterations"]
            # Step 1 reads every hub's list.
            assert e.iter_stats(1)["edges_scanned"] == int(g.outdeg[hub].sum())
