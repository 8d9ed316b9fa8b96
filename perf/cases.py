"""Performance cases: the calls a user of this package makes, over the sizes
they are made at.

A case is a dict of plain values.  ``listed()`` names twelve, ``draw(rng)``
gives another one of the same ranges, ``prepare`` makes the inputs and the
loaded engine from a seed, ``run`` is one pass through the public entry
points, ``work`` what the pass cannot do without, and ``exact`` the same
result in 64 bits by plain torch.

Graphs are seeded R-MAT (a, b, c = .57, .19, .19, self-loops and duplicates
removed) over any number of vertices: ids drawn in [0, 2^s) are scaled down to
[0, V).
"""
import math

import numpy as np
import torch

import graphee_gb300 as gx

APPS = {"pagerank": gx.APP_PAGERANK_REF, "pagerank_std": gx.APP_PAGERANK_STD, "sssp": gx.APP_SSSP,
        "sssp_weighted": gx.APP_SSSP, "cc": gx.APP_CC}
DAMPING = 0.85
RESTART = 0.15
TOLERANCE = 1e-6
DEVICE = "cuda"


def listed():
    return [
        # The smallest calls: an ego network or a test graph, where a run is launches and latency.
        {"name": "pagerank_1k", "path": "run", "app": "pagerank", "vertices": 1000, "edge_factor": 8, "shards": 4,
         "relabel": 0, "iters": 20},
        {"name": "sssp_unit_20k", "path": "run", "app": "sssp", "vertices": 20011, "edge_factor": 16, "shards": 8,
         "relabel": 0, "iters": 1000},
        # The configuration the ranks are compared at: scale 20, 256 shards, 20 supersteps.
        {"name": "pagerank_rmat20", "path": "run", "app": "pagerank", "vertices": 1 << 20, "edge_factor": 16,
         "shards": 256, "relabel": 0, "iters": 20},
        # Standard PageRank to a tolerance on a graph of no round size, in the caller's numbering.
        {"name": "pagerank_std_7m", "path": "run", "app": "pagerank_std", "vertices": 7000003, "edge_factor": 16,
         "shards": 100, "relabel": 0, "iters": 200},
        # The benchmark's headline: scale 26, relabelled at load, 20 supersteps on the resident graph.
        {"name": "pagerank_rmat26", "path": "run", "app": "pagerank", "vertices": 1 << 26, "edge_factor": 16,
         "shards": 256, "relabel": 1, "iters": 20},
        # End to end: load from host arrays, run, read the ranks back.
        {"name": "end_to_end_rmat23", "path": "load", "app": "pagerank", "vertices": 1 << 23, "edge_factor": 16,
         "shards": 256, "relabel": 0, "iters": 20},
        # Weighted SSSP, weights in [1, 255], scale 24.
        {"name": "sssp_weighted_rmat24", "path": "run", "app": "sssp_weighted", "vertices": 1 << 24,
         "edge_factor": 16, "shards": 256, "relabel": 0, "iters": 10000},
        # Connected components of a symmetrised graph.
        {"name": "cc_rmat22", "path": "run", "app": "cc", "vertices": 1 << 22, "edge_factor": 16, "shards": 256,
         "relabel": 0, "iters": 10000},
        # Triangles of a symmetrised graph.
        {"name": "triangles_rmat20", "path": "triangles", "vertices": 1 << 20, "edge_factor": 16, "shards": 256,
         "relabel": 0},
        # Personalized PageRank of 64 sources at once, the rank matrix read back.
        {"name": "ppr64_rmat20", "path": "ppr", "vertices": 1 << 20, "edge_factor": 16, "shards": 256, "relabel": 0,
         "sources": 64, "iters": 20},
        # Many independent graphs of uneven sizes in one call, PageRank and components of each.
        {"name": "batch_512", "path": "batch", "instances": 512, "scale_min": 10, "scale_max": 17, "ragged": 0,
         "iters": 30},
        # Semi-external: about half of the edges stay in the shard cache, the rest streams from host memory.
        {"name": "stream_rmat24", "path": "stream", "app": "pagerank", "vertices": 1 << 24, "edge_factor": 16,
         "shards": 256, "budget": 0.5, "iters": 10},
    ]


def draw(rng):
    path = rng.choice(["run", "run", "sssp", "cc", "load", "triangles", "ppr", "batch", "stream"])

    def vertices(lo, hi):
        return int(2.0 ** rng.uniform(lo, hi))

    shards = rng.choice([1, 8, 37, 256])
    relabel = rng.randrange(2)
    if path == "run":
        app = rng.choice(["pagerank", "pagerank", "pagerank_std"])
        return {"path": "run", "app": app, "vertices": vertices(9.5, 25), "edge_factor": rng.choice([8, 16, 16, 24]),
                "shards": shards, "relabel": relabel, "iters": 200 if app == "pagerank_std" else rng.randint(10, 30)}
    if path == "sssp":
        return {"path": "run", "app": rng.choice(["sssp", "sssp_weighted"]), "vertices": vertices(10, 24),
                "edge_factor": rng.choice([8, 16]), "shards": shards, "relabel": relabel, "iters": 10000}
    if path == "cc":
        return {"path": "run", "app": "cc", "vertices": vertices(10, 23), "edge_factor": rng.choice([4, 8, 16]),
                "shards": shards, "relabel": relabel, "iters": 10000}
    if path == "load":
        return {"path": "load", "app": "pagerank", "vertices": vertices(12, 23.5), "edge_factor": rng.choice([8, 16]),
                "shards": shards, "relabel": relabel, "iters": rng.randint(10, 30)}
    if path == "triangles":
        return {"path": "triangles", "vertices": vertices(10, 20.5), "edge_factor": rng.choice([8, 16]),
                "shards": shards, "relabel": relabel}
    if path == "ppr":
        return {"path": "ppr", "vertices": vertices(10, 20), "edge_factor": rng.choice([8, 16]), "shards": shards,
                "relabel": relabel, "sources": rng.randint(1, 64), "iters": rng.randint(10, 30)}
    if path == "batch":
        return {"path": "batch", "instances": int(2.0 ** rng.uniform(2, 9)), "scale_min": rng.randint(6, 10),
                "scale_max": rng.randint(12, 17), "ragged": 1, "iters": rng.randint(10, 40)}
    return {"path": "stream", "app": "pagerank", "vertices": vertices(18, 23.5), "edge_factor": rng.choice([8, 16]),
            "shards": rng.choice([37, 256]), "budget": round(rng.uniform(0.3, 0.8), 2), "iters": rng.randint(5, 15)}


# ---------------------------------------------------------------- inputs ----

def _rmat(sizes, edges, gen):
    """Edges of R-MAT graphs side by side: graph i has sizes[i] vertices and
    edges[i] draws.  Returns (src, dst) with each graph's first vertex added."""
    begin = np.concatenate([[0], np.cumsum(sizes)])
    levels = [max(1, math.ceil(math.log2(v))) for v in sizes]
    parts = []
    one = len(sizes) == 1
    step = 1 << 27
    total = int(sum(edges))
    if not one:
        cnt = torch.tensor(edges, device=DEVICE)
        ends = torch.cumsum(cnt, 0)
        t_lev = torch.tensor(levels, device=DEVICE)
        t_siz = torch.tensor(sizes, device=DEVICE)
        t_beg = torch.tensor(begin[:-1], device=DEVICE)
    for at in range(0, total, step):
        n = min(step, total - at)
        s = torch.zeros(n, dtype=torch.int32, device=DEVICE)
        d = torch.zeros(n, dtype=torch.int32, device=DEVICE)
        if not one:
            inst = torch.searchsorted(ends, torch.arange(at, at + n, device=DEVICE), right=True)
            lev = t_lev[inst]
        for level in range(max(levels)):
            u = torch.rand(n, device=DEVICE, generator=gen)
            sb = u >= 0.76
            db = ((u >= 0.57) & ~sb) | (u >= 0.95)
            if one:
                s = s * 2 + sb
                d = d * 2 + db
            else:
                on = lev > level
                s = torch.where(on, s * 2 + sb, s)
                d = torch.where(on, d * 2 + db, d)
        s, d = s.long(), d.long()
        if one:
            s, d = (s * sizes[0]) >> levels[0], (d * sizes[0]) >> levels[0]
        else:
            size, beg = t_siz[inst], t_beg[inst]
            s, d = ((s * size) >> lev) + beg, ((d * size) >> lev) + beg
        parts.append((s, d))
    return torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])


def _graph(case, seed):
    """(off, col, outdeg, first vertex of every graph) as device tensors; col ascending per destination."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    if case["path"] == "batch":
        r = np.random.default_rng(case["instances"])  # the sizes belong to the case, the edges to the seed
        lo, hi, n = case["scale_min"], case["scale_max"], case["instances"]
        if case["ragged"]:
            sizes = [int(2.0 ** x) for x in r.uniform(lo, hi, n)]
        else:
            sizes = [1 << int(x) for x in r.integers(lo, hi + 1, n)]
        edges = [v * int(f) for v, f in zip(sizes, r.integers(8, 33, n))]
    else:
        sizes, edges = [case["vertices"]], [case["vertices"] * case["edge_factor"]]
    V = sum(sizes)
    src, dst = _rmat(sizes, edges, gen)
    if case["path"] == "triangles" or case.get("app") == "cc":
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    key = dst * V + src
    key = key[src != dst]
    del src, dst
    key = torch.unique(key)
    dst = key // V
    col = (key - dst * V).to(torch.int32)
    del key
    off = torch.zeros(V + 1, dtype=torch.int64, device=DEVICE)
    off[1:] = torch.cumsum(torch.bincount(dst, minlength=V), 0)
    del dst
    outdeg = torch.bincount(col, minlength=V).to(torch.int32)
    first = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    return off, col, outdeg, first


def _sources(case, seed, outdeg):
    have = torch.nonzero(outdeg).reshape(-1)
    if have.numel() == 0:
        have = torch.arange(1, device=DEVICE)
    r = np.random.default_rng(seed + 1)
    pick = r.integers(0, have.numel(), case.get("sources", 1))
    return have[torch.from_numpy(pick).to(DEVICE)].cpu().numpy().astype(np.int32)


def prepare(case, seed):
    off, col, outdeg, first = _graph(case, seed)
    g = gx.Graph(off.numel() - 1, off.cpu().numpy(), col.cpu().numpy(), outdeg.cpu().numpy(), case.get("shards", 1))
    if case.get("app") == "sssp_weighted":
        gen = torch.Generator(device=DEVICE)
        gen.manual_seed(seed + 2)
        g.weights = torch.randint(1, 256, (g.E,), device=DEVICE, generator=gen,
                                  dtype=torch.int32).cpu().numpy().view(np.uint32)
    config = {"relabel": case.get("relabel", 0)}
    if case["path"] == "stream":
        config["cache_budget_bytes"] = int(case["budget"] * 4 * g.E)
    state = {"path": case["path"], "engine": gx.Engine(**config), "iters": case.get("iters", 0),
             "app": APPS.get(case.get("app")), "options": {}, "buffer": np.zeros(g.V, np.uint32)}
    if case["path"] == "load":
        state["graph"] = g
    else:
        state["engine"].load(g)
    if case.get("app") == "pagerank_std":
        state["options"] = {"tolerance": TOLERANCE}
    if case.get("app", "").startswith("sssp"):
        state["options"] = {"source": int(_sources(case, seed, outdeg)[0]), "weighted": case["app"] == "sssp_weighted"}
    if case["path"] == "ppr":
        state["sources"] = _sources(case, seed, outdeg)
    if case["path"] == "batch":
        state["first"] = first
    return state


# ------------------------------------------------------------------ pass ----

def run(state):
    e = state["engine"]
    if state["path"] == "triangles":
        return {"triangles": e.triangle_count()[0]}
    if state["path"] == "ppr":
        return {"ranks": e.ppr(state["sources"], state["iters"], RESTART)[0]}
    if state["path"] == "batch":
        pr, cc, pr_steps, cc_steps, _ = e.batch_run(state["first"], state["iters"])
        return {"ranks": pr, "labels": cc, "rank_steps": pr_steps, "label_steps": cc_steps}
    if state["path"] == "load":
        e.load(state["graph"])
    stats = e.run(state["app"], state["iters"], **state["options"])
    values = e.values(out=state["buffer"])
    if values.dtype == np.uint32:  # weighted distances, as a type that torch indexes too
        values = values.view(np.int32)
    return {"values": values, "iterations": stats["iterations"]}


def _size(case):
    if case["path"] == "batch":
        lo, hi = case["scale_min"], case["scale_max"]
        mean = (2.0 ** (hi + 1) - 2.0 ** lo) / (hi + 1 - lo)
        V = case["instances"] * mean
        return V, 20 * V
    V = case["vertices"]
    return V, V * case["edge_factor"] * (2 if case["path"] == "triangles" or case.get("app") == "cc" else 1)


def work(case):
    """Source ids once a superstep, and per vertex and superstep its offset, old value and out-degree read and its
    value and contribution written (20 bytes); SSSP, components and triangles read every edge once."""
    V, E = _size(case)
    if case["path"] == "triangles":
        return {"bytes": 4 * E + 8 * V, "flops": E}
    if case["path"] == "ppr":
        k = case["sources"]
        return {"bytes": case["iters"] * (4 * E + (8 + 8 * k) * V), "flops": 2.0 * k * E * case["iters"]}
    if case["path"] == "batch":
        return {"bytes": (case["iters"] + 5) * (4 * E + 20 * V), "flops": (case["iters"] + 5) * E}
    if case["app"] in ("sssp", "sssp_weighted", "cc"):
        return {"bytes": (8 if case["app"] == "sssp_weighted" else 4) * E + 16 * V, "flops": E}
    steps = 20 if case["app"] == "pagerank_std" else case["iters"]
    return {"bytes": steps * (4 * E + 20 * V), "flops": 2.0 * steps * E}


# ----------------------------------------------------------------- exact ----

def exact(case, seed):
    """Ranks in 64 bits by sparse products in torch; distances, labels and counts are whole numbers."""
    if case["path"] == "triangles" or case.get("app") in ("sssp", "sssp_weighted", "cc"):
        return None
    off, col, outdeg, first = _graph(case, seed)
    V = off.numel() - 1
    ones = torch.ones(col.numel(), dtype=torch.float64, device=DEVICE)
    A = torch.sparse_csr_tensor(off.to(torch.int32), col, ones, size=(V, V))
    share = 1.0 / outdeg.clamp(min=1).double()
    if case["path"] == "ppr":
        src = torch.from_numpy(_sources(case, seed, outdeg)).long().to(DEVICE)
        S = torch.zeros(V, len(src), dtype=torch.float64, device=DEVICE)
        S[src, torch.arange(len(src), device=DEVICE)] = 1.0
        R = S
        for _ in range(case["iters"]):
            R = RESTART * S + (1 - RESTART) * (A @ (R * share[:, None]))
        return {"ranks": R}
    inv_n = torch.full((V,), 1.0 / V, dtype=torch.float64, device=DEVICE)
    if case["path"] == "batch":
        sizes = torch.from_numpy(np.diff(first)).to(DEVICE)
        inv_n = torch.repeat_interleave(1.0 / sizes.double(), sizes)
    r = inv_n.clone()
    sink = (outdeg == 0).double()
    for _ in range(case["iters"]):
        acc = (A @ (r * share)[:, None]).reshape(-1)
        if case.get("app") == "pagerank_std":
            new = (1 - DAMPING) * inv_n + DAMPING * (acc + (r * sink).sum() * inv_n)
            moved = float((new - r).abs().sum())
            r = new
            if moved < TOLERANCE:
                break
        else:
            r = DAMPING * acc + inv_n
    if case["path"] == "batch":
        return {"ranks": r, "labels": None, "rank_steps": None, "label_steps": None}
    return {"values": r, "iterations": None}
