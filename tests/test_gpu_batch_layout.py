"""The rewritten instances of the batched kernel at the edges of their layout:
sizes around 16-bit ids, around the table in shared memory and of one vertex,
in-lists around a lane's, half a warp's, a warp round's and a class's length,
at any position of the first edge, against sums in 64 bits and the oracle.
"""
import numpy as np
import pytest

import graphee_gb300 as gx
import gx_oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 3, 4, 5, 31, 32, 33, 34, 60, 61, 62, 63, 64, 65, 66, 127, 128, 129, 255, 256, 257, 512, 513, 514,
           640, 1000, 8000, 8064, 8065, 9000]


def instance(n, lists, fill, rng):
    d = np.minimum(np.full(n, fill), n)
    d[:len(lists)] = np.minimum(lists, n)[:n]
    d = d[rng.permutation(n)]
    dst = np.repeat(np.arange(n), d)
    src = np.concatenate([rng.permutation(n)[:k] if k > 40 else rng.integers(0, n, k) for k in d]) if len(dst) else dst
    return gx.build_csc(n, src.astype(np.int32), dst.astype(np.int32))


@pytest.mark.parametrize("tuning", [None, dict(threads=64, lane_max=0, ctas_per_sm=4),
                                    dict(threads=512, lane_max=300, ctas_per_sm=2),
                                    dict(threads=1024, lane_max=32, ctas_per_sm=1)])
def test_layout_edges(tuning):
    rng = np.random.default_rng(7)
    parts = [(1, [], 0), (2, [2, 2], 0), (31, [], 0), (33, [33], 1), (700, LENGTHS, 2), (10007, LENGTHS * 3, 1),
             (20489, LENGTHS, 3), (65534, LENGTHS, 1), (65535, LENGTHS * 2, 1), (65536, LENGTHS, 0),
             (70001, LENGTHS, 2)]
    offs, cols, vb, base = [], [], [0], 0
    for n, lists, fill in parts:
        off, col = instance(n, lists, fill, rng)
        offs.append(off[:-1] + base)
        cols.append(col + vb[-1])
        base += int(off[-1])
        vb.append(vb[-1] + n)
    g = gx.Graph(vb[-1], np.concatenate(offs + [[base]]), np.concatenate(cols), None, 1)
    with gx.Engine() as e:
        e.load(g)
        pr, cc, ps, cs, _ = e.batch_run(np.array(vb, np.int32), pr_iters=12, cc_max_iter=1000, tuning=tuning)
    for i, (n, _, _) in enumerate(parts):
        b, off = vb[i], g.off[vb[i]:vb[i + 1] + 1] - g.off[vb[i]]
        col, od = g.col[g.off[b]:g.off[vb[i + 1]]] - b, g.outdeg[b:vb[i + 1]]
        dst = np.repeat(np.arange(n), np.diff(off))
        r = np.full(n, 1.0 / n)
        for _ in range(ps[i]):
            r = 0.85 * np.bincount(dst, (r / np.maximum(od, 1))[col], n) + 1.0 / n
        # FP32 sums of positive terms of at most 9000 edges, in lane sums and trees: the parity bound.
        assert np.max(np.abs(pr[b:b + n] - r) / r) < 1e-5, n
        ref, changed, _ = O.run(O.CC, n, 1, np.array([0, n], np.int32), off, col, od, 1000)
        assert np.array_equal(cc[b:b + n], ref), n
        assert cs[i] == len(changed), n
