"""Batches whose preparation is shared out differently: instances sorted by a
CTA or by several, checked and written out by one to hundreds, tiny ones by the
wave, one long instance among many short ones; against the oracle, and the same
bits by every schedule.
"""
import numpy as np
import pytest

import graphee_gb300 as gx
import gx_oracle as O

pytestmark = pytest.mark.gpu


def packed(sizes, seed):
    """Graphs of the given vertex counts side by side: random edges, a hub with a long list, some without edges."""
    rng = np.random.default_rng(seed)
    vb = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    m = np.where(rng.random(len(sizes)) < 0.1, 0, 6 * np.array(sizes))
    inst = np.repeat(np.arange(len(sizes)), m)
    n = np.array(sizes)[inst]
    src = vb[inst] + (rng.random(len(inst)) ** 2 * n).astype(np.int64)
    dst = vb[inst] + np.where(rng.random(len(inst)) < 0.3, 0, (rng.random(len(inst)) * n).astype(np.int64))
    off, col = gx.build_csc(int(vb[-1]), src, dst)
    return gx.Graph(int(vb[-1]), off, col, None, 1), vb


CASES = {
    "one, a CTA": [2048], "one, several": [2049], "one, wide ids": [70001], "few": [5000, 33000, 2, 9000, 1],
    "one long among many": [40] * 200 + [33000] + [300] * 200, "as many as SMs": [2500] * 152, "fewer than SMs": [2500] * 151,
    "tiny, in waves": [1 + i % 256 for i in range(1300)], "tiny, few": [256] * 9, "very many": [1 + i % 4 for i in range(70000)],
    "very many and a long one": [2] * 66000 + [40000],
}


@pytest.mark.parametrize("name", CASES)
def test_against_oracle(name):
    sizes = CASES[name]
    g, vb = packed(sizes, len(sizes))
    with gx.Engine() as e:
        e.load(g)
        pr, cc, ps, cs, _ = e.batch_run(vb, 12, 1000)
        for tuning in ({"threads": 512, "ctas_per_sm": 2}, {"threads": 64, "ctas_per_sm": 16}):
            for x, y in zip((pr, cc, ps, cs), e.batch_run(vb, 12, 1000, tuning=tuning)):
                assert np.array_equal(x, y)
    order = np.argsort(np.diff(g.off[vb]))
    for i in set(order[[0, len(order) // 2, -2 if len(order) > 1 else -1, -1]].tolist()):
        b, t = int(vb[i]), int(vb[i + 1])
        off, col, od = g.off[b:t + 1] - g.off[b], g.col[g.off[b]:g.off[t]] - b, g.outdeg[b:t]
        a = (t - b, 1, np.array([0, t - b], np.int32), off, col, od)
        exact = np.full(t - b, 1.0 / (t - b))
        at = np.repeat(np.arange(t - b), np.diff(off))
        for _ in range(ps[i]):
            exact = 0.85 * np.bincount(at, (exact / np.maximum(od, 1))[col], t - b) + 1.0 / (t - b)
        assert np.max(np.abs(pr[b:t] - exact) / exact) < 1e-5, i
        assert ps[i] == len(O.run(O.PAGERANK_REF, *a, 12)[1]), i
        labels, changed, _ = O.run(O.CC, *a, 1000)
        assert np.array_equal(cc[b:t], labels) and cs[i] == len(changed), i
