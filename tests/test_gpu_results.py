"""Results in the caller's memory, of every kind that it may have: fresh pages,
pages in use, an odd start, pinned memory; below, at and above the size from
which they travel in pinned pieces (128 MB).
"""
import numpy as np
import pytest

import graphee_gb300 as gx

pytestmark = pytest.mark.gpu

STAGE = 1 << 25  # 4-byte values


@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("V", [1, 16389, STAGE - 1, STAGE, STAGE + 2097153])
def test_values_arrive(V, relabel):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(V)
    src, dst = rng.integers(0, V, 64).astype(np.int32), rng.integers(0, V, 64).astype(np.int32)
    off, col = gx.build_csc(V, src, dst)
    g = gx.Graph(V, off, col, None, min(V, 3))
    start = rng.integers(0, 1 << 20, V).astype(np.float32)
    with gx.Engine(relabel=relabel) as e:
        e.load(g)
        e.set_init(start)
        e.run(gx.APP_PAGERANK_REF, 1, use_init=True)
        want = e.values()
        exact = np.full(V, 1.0 / V)
        u = np.repeat(np.arange(V), np.diff(off))
        np.add.at(exact, u, 0.85 * start[col].astype(np.float64) / np.maximum(g.outdeg, 1)[col])
        np.testing.assert_allclose(want, exact, rtol=1e-5)
        used = np.full(V, 7, np.float32)
        odd = np.full(V + 1, 7, np.float32)
        pinned = torch.full((V,), 7.0, dtype=torch.float32, pin_memory=True).numpy()
        for out in (used, odd[1:], pinned):
            e.values(out=out)
            np.testing.assert_array_equal(out, want)
        assert odd[0] == 7
