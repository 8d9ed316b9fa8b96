"""How a graph is cut into work units (unit_caps): the caller's heavy_degree and
tile_edges are obeyed at every size of graph, on the CPU; and with a bound above
the default, long lists that a tile's warp then sweeps whole, against the oracle.
"""
import subprocess

import numpy as np
import pytest

import graphee_gb300 as gx
import gx_oracle as O
from graphee_gb300 import _build

SIZES = [0, 1000, 1 << 20, 1 << 24, 30_000_000, 1 << 26, 1 << 30, 1 << 36]
HEAVY = [1, 32, 300, 512, 4095, 4096, 4097, 8192, 8193, 20000, 2**31 - 1]
TILE = [1, 32, 63, 64, 2048, 5000]
WARPS = 4864


@pytest.fixture(scope="module")
def caps(tmp_path_factory):
    d = tmp_path_factory.mktemp("caps")
    (d / "caps.cu").write_text('''
#include <cstdio>
#include <cstdlib>
#include "gx_kernels.cuh"
int main() {
  long long E;
  int heavy, tile;
  while (scanf("%lld %d %d", &E, &heavy, &tile) == 3) {
    const gx::UnitCaps c = gx::unit_caps(E, WARPS, tile, heavy);
    printf("%d %d %d\\n", c.tile, c.chunk, c.heavy);
  }
}
''')
    subprocess.run([_build.NVCC, *_build.ARCH, "-std=c++17", f"-DWARPS={WARPS}", "-I", str(_build.CSRC), "-o",
                    str(d / "caps"), str(d / "caps.cu")], check=True, capture_output=True)
    asked = [(E, h, t) for E in SIZES for h in HEAVY for t in TILE]
    out = subprocess.run([str(d / "caps")], input="".join("%d %d %d\n" % x for x in asked), text=True,
                         capture_output=True, check=True).stdout
    return {x: tuple(map(int, line.split())) for x, line in zip(asked, out.splitlines())}


def test_bounds(caps):
    assert len(caps) == len(SIZES) * len(HEAVY) * len(TILE)
    for (E, heavy, tile), (t, chunk, h) in caps.items():
        assert 32 <= t <= max(tile, 32)
        assert 256 <= chunk <= 4096 and chunk % 256 == 0
        assert 32 <= h <= max(heavy, 32)
        if heavy > 4096:
            assert h == heavy  # obeyed upwards
        elif heavy <= 512:
            assert h == max(heavy, 32)
        else:
            assert h == min(heavy, 2 * chunk)
        if E >= 60_000_000 and tile >= 64:
            assert chunk == 4096 and h == max(heavy, 32)


@pytest.mark.gpu
@pytest.mark.parametrize("relabel", [0, 1])
@pytest.mark.parametrize("heavy", [5000, 20000, 100000])
def test_long_lists_below_the_bound(heavy, relabel):
    V = 60007
    rng = np.random.default_rng(heavy)
    lists = [4096, 4097, 4999, 5000, 5001, 19999, 20001, 60000]
    dst = np.concatenate([np.repeat(np.arange(len(lists)), lists), rng.integers(0, V, 2 * V)])
    src = np.concatenate([rng.permutation(V)[:n] for n in lists] + [rng.integers(0, V, 2 * V)])
    off, col = gx.build_csc(V, src, dst)
    g = gx.Graph(V, off, col, None, 5)
    g.weights = gx.edge_weights(4, g)
    a = (g.V, g.P, g.bounds, g.off, g.col, g.outdeg)
    at = np.repeat(np.arange(V), np.diff(g.off))
    exact = np.full(V, 1.0 / V)
    for _ in range(8):
        exact = 0.85 * np.bincount(at, (exact / np.maximum(g.outdeg, 1))[g.col], V) + 1.0 / V
    with gx.Engine(relabel=relabel, heavy_degree=heavy) as e:
        e.load(g)
        e.run(gx.APP_PAGERANK_REF, 8)
        assert np.max(np.abs(e.values().astype(np.float64) - exact) / exact) < 1e-5
        e.run(gx.APP_CC, 1000)
        assert np.array_equal(e.values(), O.run(O.CC, *a, 1000)[0])
        e.run(gx.APP_SSSP, 1000, source=3, weighted=True)
        assert np.array_equal(e.values(), O.run(O.SSSP, *a, 1000, weights=g.weights, source=3)[0])
