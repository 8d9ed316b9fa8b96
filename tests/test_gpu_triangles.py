"""Triangle counts at the edges of the counting kernels: graphs around the
bitmap's least size (ids, or ranks with vertices below the bitmap), cores at
either end of the ids, list lengths around 16-byte pieces and a half-warp's
64 entries, and more than one hash table of out-neighbours.
"""
import numpy as np
import pytest

import graphee_gb300 as gx
import gx_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("V", [3, 33, 5000, (1 << 18) - 1, 1 << 18, (1 << 18) + 1, 300007])
def test_triangles_edges(V, relabel):
    rng = np.random.default_rng(V)
    src, dst = [rng.integers(0, V, 2 * V)], [rng.integers(0, V, 2 * V)]
    # Cliques of sizes around the pieces, at the low and high end of the ids and spread over them.
    at = 0
    for k in [2, 3, 4, 5, 8, 9, 17, 33, 62, 65, 66, 129, 130, 257]:
        for ids in (np.arange(at, at + k), V - 1 - np.arange(at, at + k), rng.integers(0, V, k)):
            ids = ids[(ids >= 0) & (ids < V)]
            a, b = np.meshgrid(ids, ids)
            src.append(a.ravel())
            dst.append(b.ravel())
        at += k // 2
    # A hub next to everything.
    src.append(np.full(V, V // 2))
    dst.append(np.arange(V))
    off, col = gx.build_csc(V, np.concatenate(src), np.concatenate(dst),
                            gx.BUILD_DROP_SELF | gx.BUILD_DEDUP | gx.BUILD_SYMMETRIZE)
    g = gx.Graph(V, off, col, None, min(5, V))
    with gx.Engine(relabel=relabel) as e:
        e.load(g)
        assert e.triangle_count()[0] == O.triangles(V, off, col)
        assert e.triangle_count()[0] == O.triangles(V, off, col)


def test_triangles_long_lists_below_the_bitmap():
    """Circulant graph C_V(1..k): V k (k - 1) / 2 triangles.  All degrees are equal, so the lowest ids lie below the
    bitmap with out-lists of up to 2k entries, more than one of a warp's tables."""
    V, k = (1 << 18) + 700, 400
    near = np.concatenate([np.arange(-k, 0), np.arange(1, k + 1)])
    col = np.sort((np.arange(V, dtype=np.int32)[:, None] + near[None, :].astype(np.int32)) % V, axis=1)
    g = gx.Graph(V, np.arange(V + 1, dtype=np.int64) * (2 * k), col.reshape(-1), np.full(V, 2 * k, np.int32), 1)
    with gx.Engine() as e:
        e.load(g)
        assert e.triangle_count()[0] == V * k * (k - 1) // 2
