"""Personalized PageRank at the edges of its work units: in-lists around a
stream's batch, the chunked length and the chunk, runs between chunked
vertices, every row width, both layouts, against sums in 64 bits.
"""
import numpy as np
import pytest

import graphee_gb300 as gx
import gx_oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 7, 8, 9, 255, 256, 257, 511, 512, 513, 514, 767, 768, 769, 2000, 0, 9000, 513, 1, 600]


@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("V,fill", [(1, 0), (40, 2), (12011, 1), (60013, 3)])
@pytest.mark.parametrize("k", [1, 9, 20, 64])
def test_ppr_units(k, V, fill, relabel):
    rng = np.random.default_rng(V + k)
    n = np.full(V, fill)
    at = np.arange(0, V, max(1, V // 200))[:200]
    n[at] = np.array(LENGTHS * 10)[:len(at)]
    n = np.minimum(n, V)
    dst = np.repeat(np.arange(V), n)
    src = np.concatenate([rng.permutation(V)[:d] if d > fill else rng.integers(0, V, d) for d in n]) if n.sum() else dst
    off, col = gx.build_csc(V, src, dst)
    g = gx.Graph(V, off, col, None, min(3, V))
    sources = rng.integers(0, V, k).astype(np.int32)
    with gx.Engine(relabel=relabel) as e:
        e.load(g)
        R, st = e.ppr(sources, 9)
        again, _ = e.ppr(sources, 9)
        none, _ = e.ppr(sources, 0)
    assert np.array_equal(R, again)
    # FP32 sums of terms that add up to at most 1: the parity bound of the existing test.
    assert np.abs(R - O.ppr(V, g.off, g.col, g.outdeg, sources, 9, 0.15)).max() < 1e-6
    assert np.array_equal(none, np.eye(V, dtype=np.float32)[:, sources] if V <= 40 else
                          (np.arange(V)[:, None] == sources[None, :]).astype(np.float32))
