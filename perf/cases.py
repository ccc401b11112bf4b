"""Workloads of the traversal library as its users run them, for timing and comparing builds.

A case is a dict of plain values: `op` (the entry points called), the graph (`graph`, `V`, `E`), the number of
`sources`, the SSSP `delta` (0 = Bellman-Ford), the `schedule` (plain or learned) and where results go (`out`).
Graphs are drawn on the GPU from the seed alone: RMAT edges with a/b/c/d 57/19/19/5 percent and weights in [0, 1],
uniform random edges with weights in [0, 1), or a 4-neighbour grid with integer weights in [1, 100); self-loops are
dropped, except for the optimisation pass, whose work that is.  V need not be a power of two.

Distances are returned twice, as floats and as the same memory read as integers: the library promises the
reference's fp32 bits, and the sentinel of unreachable vertices (FLT_MAX) would hide a wrong distance in a norm.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parallel-task1_b200"))

import pytrav as T  # noqa: E402
from pytrav import learn  # noqa: E402

FLT_MAX = float(np.finfo(np.float32).max)
BIG = 270_000_000  # most edges of a case: the RMAT scale 23, edge factor 32 benchmark graph


def listed():
    return [
        # the smallest call: one BFS on a graph of a thousand vertices; launches and host work are all of it
        dict(name="bfs_small", op="query", kinds="bfs", graph="rmat", V=1 << 10, E=8 << 10, sources=1, delta=0.0,
             schedule="plain", out="device"),
        # the reference's own configuration: Bellman-Ford from one source, RMAT scale 16, edge factor 16, results
        # copied to the host as the sample program has them
        dict(name="sssp_s16_host", op="query", kinds="sssp", graph="rmat", V=1 << 16, E=1 << 20, sources=1, delta=0.0,
             schedule="plain", out="host"),
        # an even-degree random graph of an odd size, BFS and delta-stepping from two sources
        dict(name="uniform_1m", op="query", kinds="both", graph="uniform", V=1_000_003, E=16_000_000, sources=2,
             delta=0.1, schedule="plain", out="device"),
        # a road-like graph of high diameter, ragged sides; delta tuned to its weights (6.4 x mean weight / degree)
        dict(name="grid_1m", op="query", kinds="both", graph="grid", V=1100 * 911, E=4 * 1100 * 911, sources=1,
             delta=80.0, schedule="plain", out="device"),
        # the benchmark's graph size (RMAT scale 23, edge factor 32), single queries: BFS with Beamer's switch and
        # SSSP with the learned schedule
        dict(name="bfs_s23", op="query", kinds="bfs", graph="rmat", V=1 << 23, E=32 << 23, sources=4, delta=0.0,
             schedule="plain", out="device"),
        dict(name="sssp_s23", op="query", kinds="sssp", graph="rmat", V=1 << 23, E=32 << 23, sources=1, delta=0.1,
             schedule="learned", out="device"),
        # many queries over many small graphs in one launch: 64 graphs of scales 10-18, 512 queries
        dict(name="batch_many", op="batch", kinds="both", graph="rmat", V=0, E=0, graphs=64, sources=8, delta=0.1,
             schedule="plain", out="device", team=8),
        # the benchmark's end-to-end step, smaller: BFS and SSSP from 16 sources of one graph in one batch, results
        # in pinned host memory
        dict(name="batch_host_s21", op="batch", kinds="both", graph="rmat", V=1 << 21, E=32 << 21, graphs=1,
             sources=16, delta=0.1, schedule="learned", out="host", team=74),
        # the reference's wrappers on device edge lists, as its own callers and transitive closure call them
        dict(name="el_bfs_s20", op="el_bfs", graph="rmat", V=1 << 20, E=16 << 20),
        dict(name="el_sssp_300k", op="el_sssp", graph="rmat", V=300_007, E=4_800_000),
        # a graph loaded from a file: host edge arrays to a device graph, then one BFS and one SSSP to the host
        dict(name="load_query_s18", op="load", graph="rmat", V=1 << 18, E=16 << 18, delta=0.1),
        # the optimisation pass before a graph is stored: duplicates and loops out, cache-segment order
        dict(name="optimize_s19", op="optimize", graph="rmat", V=1 << 19, E=16 << 19, segment=1 << 17),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["query", "query", "query", "query", "batch", "batch", "el_bfs", "el_sssp", "load", "optimize"])
    V = _log(rng, 1000, 1 << 21)
    E = V * rng.randint(8, 32)
    if op in ("el_bfs", "el_sssp", "load", "optimize"):
        V = _log(rng, 1000, 1 << 20)
        c = dict(op=op, graph=rng.choice(["rmat", "rmat", "uniform"]), V=V, E=V * rng.randint(8, 16))
        if op == "load":
            c["delta"] = rng.choice([0.05, 0.1, 0.2])
        if op == "optimize":
            c["segment"] = rng.choice([0, V // 4 + 1])
        return c
    if op == "batch":
        many = rng.random() < 0.5
        c = dict(op="batch", kinds="both", graph="rmat", V=0 if many else V, E=0 if many else E,
                 graphs=rng.randint(8, 64) if many else 1, sources=rng.randint(2, 8) if many else rng.randint(4, 16),
                 delta=rng.choice([0.05, 0.1, 0.2]), schedule=rng.choice(["plain", "learned"]),
                 out=rng.choice(["device", "host"]))
        c["team"] = 8 if many or V < 100_000 else 74
        return c
    c = dict(op="query", kinds=rng.choice(["bfs", "sssp", "both"]),
             graph=rng.choice(["rmat", "rmat", "uniform", "grid"]), V=V, E=E, sources=rng.randint(1, 4),
             delta=rng.choice([0.0, 0.05, 0.1, 0.2]), schedule=rng.choice(["plain", "learned"]),
             out=rng.choice(["device", "device", "host"]))
    if c["graph"] == "rmat" and rng.random() < 0.3:  # the large single graphs
        c["V"] = _log(rng, 1 << 21, 1 << 23)
        c["E"] = min(c["V"] * rng.randint(8, 32), BIG)
    if c["graph"] == "grid":
        a = max(2, int(math.sqrt(V) * rng.uniform(0.7, 1.4)))
        c["V"], c["delta"] = a * max(2, V // a), 80.0
        c["E"], c["sources"] = 4 * c["V"], 1
    if c["delta"] == 0.0:
        c["schedule"] = "plain"  # the learned schedule needs a finite delta
    return c


# ------------------------------------------------------------------ graphs
def _grid_sides(V):
    a = int(math.isqrt(V))
    while V % a:
        a -= 1
    return V // a, a


def _edges(kind, V, E, seed, loops=False):
    """(src, dst, w) on the GPU; self-loops are dropped unless `loops`."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    dev = dict(device="cuda")
    if kind == "grid":
        h, wd = _grid_sides(V)
        idx = torch.arange(V, dtype=torch.int32, **dev).view(h, wd)
        pairs = [(idx[:, :-1], idx[:, 1:]), (idx[:, 1:], idx[:, :-1]), (idx[:-1], idx[1:]), (idx[1:], idx[:-1])]
        src = torch.cat([a.reshape(-1) for a, _ in pairs])
        dst = torch.cat([b.reshape(-1) for _, b in pairs])
        w = torch.randint(1, 100, (src.numel(),), generator=g, **dev).float()
        return src, dst, w
    if kind == "uniform":
        src = torch.randint(0, V, (E,), generator=g, dtype=torch.int32, **dev)
        dst = torch.randint(0, V, (E,), generator=g, dtype=torch.int32, **dev)
    else:
        scale = max(1, (V - 1).bit_length())
        src = torch.zeros(E, dtype=torch.int32, **dev)
        dst = torch.zeros(E, dtype=torch.int32, **dev)
        for _ in range(scale):
            r = torch.rand(E, generator=g, **dev)
            src.mul_(2).add_(r >= 0.76)
            dst.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        if V != 1 << scale:
            src = ((src.long() * V) >> scale).int()
            dst = ((dst.long() * V) >> scale).int()
    w = torch.rand(E, generator=g, **dev)
    if loops:
        return src, dst, w
    keep = src != dst
    return src[keep], dst[keep], w[keep]


def _many(case):
    """Vertex and edge counts of a batch's graphs."""
    if case["graphs"] == 1:
        return [(case["V"], case["E"])]
    rng = np.random.default_rng(1001)
    return [(1 << int(rng.integers(10, 19)), int(rng.integers(8, 33))) for _ in range(case["graphs"])]


def _graph_edges(case, seed):
    """Edge lists of the case's graphs, in order."""
    if case["op"] != "batch":
        yield case["V"], _edges(case["graph"], case["V"], case["E"], seed, loops=case["op"] == "optimize")
        return
    for i, (V, e) in enumerate(_many(case)):
        yield V, _edges(case["graph"], V, e if case["graphs"] == 1 else V * e, seed * 101 + i)


def _sources(V, src, n, seed):
    """n distinct vertices with out-edges."""
    cand = torch.unique(src).cpu().numpy()
    rng = np.random.default_rng(seed)
    return rng.choice(cand, size=min(n, len(cand)), replace=False).astype(np.int32)


# ----------------------------------------------------------------- prepare
def _empty(shape, dtype, host):
    return torch.empty(shape, dtype=dtype).pin_memory() if host else torch.empty(shape, dtype=dtype, device="cuda")


def prepare(case, seed):
    op = case["op"]
    s = dict(case=case)
    if op == "query":
        (V, (src, dst, w)), = _graph_edges(case, seed)
        srcs = _sources(V, src, case["sources"], seed)
        torch.cuda.synchronize()
        g = T.Graph.from_edges(V, src, dst, w)
        if case["schedule"] == "learned":
            learn.install(g, delta=case["delta"])
        host, n = case["out"] == "host", len(srcs)
        s.update(g=g, sources=srcs, sched=T.SCHEDULE_LEARNED if case["schedule"] == "learned" else T.SCHEDULE_PLAIN)
        if case["kinds"] != "sssp":
            s["levels"] = _empty((n, V), torch.int32, host)
        if case["kinds"] != "bfs":
            s["dist"] = _empty((n, V), torch.float32, host)
    elif op == "batch":
        graphs, picks = [], []
        for i, (V, (src, dst, w)) in enumerate(_graph_edges(case, seed)):
            picks.append(_sources(V, src, case["sources"], seed + i))
            torch.cuda.synchronize()
            g = T.Graph.from_edges(V, src, dst, w)
            if case["schedule"] == "learned":
                learn.install(g, delta=case["delta"])
            graphs.append(g)
        host = case["out"] == "host"
        sched = T.SCHEDULE_LEARNED if case["schedule"] == "learned" else T.SCHEDULE_PLAIN
        # one graph: BFS and SSSP from every source; many graphs: the sources alternate between the two
        todo = [(gi, kind, int(x)) for gi, p in enumerate(picks) for k, x in enumerate(p)
                for kind in ((0, 1) if case["graphs"] == 1 else (k % 2,))]
        size = [sum(graphs[gi].V for gi, kind, _ in todo if kind == want) for want in (0, 1)]
        s["levels"], s["dist"] = _empty(size[0], torch.int32, host), _empty(size[1], torch.float32, host)
        at, queries = [0, 0], []
        for gi, kind, x in todo:
            V = graphs[gi].V
            out = (s["levels"], s["dist"])[kind][at[kind]:at[kind] + V]
            at[kind] += V
            queries.append((gi, kind, x, case["delta"] if kind else 0.0, sched, out))
        b = T.Batch(graphs)
        b.shape = (case["team"], 32, 128) if case["team"] == 8 else (case["team"], 64, 256)
        s.update(batch=b, queries=queries, host=host)
    else:
        (V, (src, dst, w)), = _graph_edges(case, seed)
        s["source"] = int(_sources(V, src, 1, seed)[0])
        if op == "load":
            s.update(src=src.cpu().numpy(), dst=dst.cpu().numpy(), w=w.cpu().numpy())
        else:
            s.update(src=src, dst=dst, w=w)
            s["visited"] = torch.empty(V, dtype=torch.uint8, device="cuda")
            s["d"] = torch.empty(V, dtype=torch.float32, device="cuda")
    return s


# --------------------------------------------------------------------- run
def run(s):
    case = s["case"]
    op, V = case["op"], case["V"]
    if op == "query":
        out = {}
        if "levels" in s:
            out["levels"] = s["g"].bfs(s["sources"], out=s["levels"], schedule=s["sched"])
        if "dist" in s:
            dist = s["g"].sssp(s["sources"], out=s["dist"], delta=case["delta"], schedule=s["sched"])
            out.update(dist=dist, dist_bits=dist.view(torch.int32))
        return out
    if op == "batch":
        if s["host"]:
            s["batch"].run_host(s["queries"])
        else:
            s["batch"].run(s["queries"])
        return {"levels": s["levels"], "dist": s["dist"], "dist_bits": s["dist"].view(torch.int32)}
    if op == "el_bfs":
        T.bfs_wrapper(s["src"], s["dst"], V, len(s["src"]), s["visited"], s["source"])
        return {"visited": s["visited"]}
    if op == "el_sssp":
        T.init_distances(s["d"], V, s["source"])
        T.bellman_ford_wrapper(s["src"], s["dst"], s["w"], V, len(s["src"]), s["source"], s["d"])
        return {"dist": s["d"], "dist_bits": s["d"].view(torch.int32)}
    if op == "load":
        g = T.Graph.from_edges(V, s["src"], s["dst"], s["w"])
        levels = g.bfs([s["source"]])
        dist = g.sssp([s["source"]], delta=case["delta"])
        g.free()
        return {"levels": levels, "dist": dist, "dist_bits": dist.view(np.int32)}
    # the pass works in place, so the caller's edge list is copied first
    src, dst, w = s["src"].clone(), s["dst"].clone(), s["w"].clone()
    n = T.el_optimize(src, dst, w, V, case["segment"])
    for x in (src, dst, w):
        x[n:].zero_()
    return {"edges": n, "src": src, "dst": dst, "w": w}


# -------------------------------------------------------------------- work
def work(case):
    """Each input read once and each output written once: a BFS needs the row offsets and the neighbours (4 V + 4 E)
    and writes 4 V; an SSSP reads the weights too.  An edge list is 8 or 12 bytes an edge."""
    V, E, op = case["V"], case["E"], case["op"]
    if op == "el_bfs":
        return {"bytes": 8 * E + V, "flops": 0}
    if op == "el_sssp":
        return {"bytes": 12 * E + 8 * V, "flops": E}
    if op == "load":
        return {"bytes": 12 * E + 8 * V, "flops": E}
    if op == "optimize":
        return {"bytes": 24 * E, "flops": 0}
    bfs, sssp = lambda V, E: 8 * V + 4 * E, lambda V, E: 8 * V + 8 * E  # noqa: E731
    if op == "query":
        b = (bfs(V, E) if case["kinds"] != "sssp" else 0) + (sssp(V, E) if case["kinds"] != "bfs" else 0)
        return {"bytes": case["sources"] * b, "flops": case["sources"] * E if case["kinds"] != "bfs" else 0}
    if case["graphs"] == 1:
        return {"bytes": case["sources"] * (bfs(V, E) + sssp(V, E)), "flops": case["sources"] * E}
    # means over scales 10-18 and edge factors 8-32; half of the queries are of each kind
    V = sum(1 << k for k in range(10, 19)) / 9
    q = case["graphs"] * case["sources"] / 2
    return {"bytes": q * (bfs(V, 20 * V) + sssp(V, 20 * V)), "flops": q * 20 * V}


# ------------------------------------------------------------------- exact
def _dist64(V, src, dst, w, sources):
    """Distances from each source in 64 bits: Bellman-Ford over the edges of the vertices that changed."""
    n = len(sources)
    d = torch.full((n, V), math.inf, dtype=torch.float64, device="cuda")
    for k, x in enumerate(sources):
        row = d[k]
        row[int(x)] = 0.0
        active = torch.zeros(V, dtype=torch.bool, device="cuda")
        active[int(x)] = True
        while True:
            e = active[src].nonzero().view(-1)
            if not e.numel():
                break
            s, t = src[e], dst[e].long()
            cand = row[s] + w[e]
            better = cand < row[t]
            t, cand = t[better], cand[better]
            if not t.numel():
                break
            old = row.clone()
            row.scatter_reduce_(0, t, cand, "amin")
            active = row < old
    return torch.where(torch.isinf(d), torch.full_like(d, FLT_MAX), d)


def exact(case, seed):
    op = case["op"]
    if op in ("el_bfs", "optimize") or case.get("kinds") == "bfs":
        return None  # whole numbers, or the inputs' own values
    dist = []
    for i, (V, (src, dst, w)) in enumerate(_graph_edges(case, seed)):
        n = case.get("sources", 1)
        srcs = _sources(V, src, n, seed + i if op == "batch" else seed)
        if op == "batch" and case["graphs"] > 1:
            srcs = srcs[1::2]
        if len(srcs):
            dist.append(_dist64(V, src, dst, w, srcs))
    if op == "batch":
        return {"levels": None, "dist": torch.cat([x.reshape(-1) for x in dist]), "dist_bits": None}
    d = dist[0]
    if op == "el_sssp":
        return {"dist": d[0], "dist_bits": None}
    return dict({"levels": None} if op == "load" or case["kinds"] == "both" else {}, dist=d, dist_bits=None)
