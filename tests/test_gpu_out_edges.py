"""The out-edge CSR by one pass and by buckets on both sides of the rule between
them: evenly spread edges that L2 holds or not, a source just below and at the
degree from which its atomics decide.  Weighted distances and labels depend on
every out-edge.
"""
import numpy as np
import pytest

import graphee_gb300 as gx
import gx_oracle as O

pytestmark = pytest.mark.gpu

CASES = {"even": (100003, 5 << 20, 0), "even, more than L2 holds": (1200007, 17 << 20, 0), "one bucket, dense": (3001, 8_000_000, 0),
         "a source below": (70001, 5 << 20, 16383), "a source at": (70001, 5 << 20, 16384), "few edges": (70001, 4_000_000, 30000)}


@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("name", CASES)
def test_both_builds(name, relabel):
    V, n, hub = CASES[name]
    rng = np.random.default_rng(V + n)
    src, dst = rng.integers(1 if hub else 0, V, n), rng.integers(0, V, n)
    if hub:
        src, dst = np.concatenate([src, np.zeros(hub, np.int64)]), np.concatenate([dst, 1 + rng.permutation(V - 1)[:hub]])
    off, col = gx.build_csc(V, src, dst)
    g = gx.Graph(V, off, col, None, 9)
    assert g.outdeg[0] == hub or not hub
    g.weights = gx.edge_weights(2, g)
    a = (g.V, g.P, g.bounds, g.off, g.col, g.outdeg)
    with gx.Engine(relabel=relabel, push_edge_fraction=1.0) as e:
        e.load(g)
        st = e.run(gx.APP_CC, 1000)
        assert st["push_iterations"] > 0
        assert np.array_equal(e.values(), O.run(O.CC, *a, 1000)[0])
        st = e.run(gx.APP_SSSP, 1000, source=V - 2, weighted=True)
        assert st["push_iterations"] == st["iterations"]
        assert np.array_equal(e.values(), O.run(O.SSSP, *a, 1000, weights=g.weights, source=V - 2)[0])
