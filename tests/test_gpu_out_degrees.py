"""Out-degrees that sum to the edges but do not count them (a vertexout.npy of
another graph): the out-edge CSR is refused, whichever kernel builds it, before
any kernel follows its entries; runs that need none of it are unaffected.
"""
import numpy as np
import pytest

import graphee_gb300 as gx
import gx_oracle as O

pytestmark = pytest.mark.gpu


def graph(V, E):
    rng = np.random.default_rng(V)
    # Source 1 in several slices of its bucket where there are that many edges.
    src = np.concatenate([rng.integers(0, V, E), np.full(V, 1), [V - 1]])
    dst = np.concatenate([rng.integers(0, V, E), np.arange(V), [0]])
    off, col = gx.build_csc(V, src, dst)
    return gx.Graph(V, off, col, None, 4)


WRONG = {"next to each other": lambda V: (2, 3), "in two buckets": lambda V: (2, V - 1), "last to first": lambda V: (V - 1, 2),
         "the hub's": lambda V: (1, 2)}


@pytest.mark.parametrize("how", WRONG)
@pytest.mark.parametrize("V,E", [(3000, 20000), (70001, 5 << 20)])
def test_refused_and_recovered(V, E, how):
    g = graph(V, E)
    a, b = WRONG[how](V)
    od = g.outdeg.copy()
    od[b] += od[a]
    od[a] = 0
    wrong = gx.Graph(V, g.off, g.col, od, g.P, g.bounds)
    with gx.Engine() as e:
        e.load(wrong)
        for app in (gx.APP_SSSP, gx.APP_CC):
            for _ in range(2):
                with pytest.raises(gx.GxError) as ei:
                    e.run(app, 100, source=0)
                assert ei.value.status == gx.GX_ERR_FORMAT
        e.load(g)
        e.run(gx.APP_SSSP, 100, source=1)
        assert np.array_equal(e.values(), O.run(O.SSSP, V, g.P, g.bounds, g.off, g.col, g.outdeg, 100, source=1)[0])
    # Without push steps nothing needs the CSR; selective PageRank steps go without its marks.
    with gx.Engine(push_sparse=0) as e:
        e.load(wrong)
        e.run(gx.APP_CC, 100)
        assert np.array_equal(e.values(), O.run(O.CC, V, g.P, g.bounds, g.off, g.col, g.outdeg, 100)[0])
    with gx.Engine(selective_threshold=2.0, exact_order=1) as e:
        e.load(wrong)
        e.run(gx.APP_PAGERANK_REF, 20)
        ref = O.run(O.PAGERANK_REF, V, g.P, g.bounds, g.off, g.col, od, 20)[0]
        assert np.array_equal(e.values().view(np.uint32), ref.view(np.uint32))
