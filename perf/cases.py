"""Performance cases: the calls that a user of the engine makes, with the
inputs those calls meet, over the sizes that the tests, the benchmark and
the library's generators use.

A case names an entry point of kites_b200.capi (``kind``), a generated graph
(``graph``, ``n``, ``m``) and the options of the call.  Graphs are made on
the GPU from the seed: R-MAT with a,b,c,d = 0.57,0.19,0.19,0.05 (the
benchmark's; ids taken modulo n, self-loops moved to the next vertex),
Erdos-Renyi, the four-neighbour grid, and disjoint unions of R-MAT graphs of
uneven size.  Weights are uniform in [1, 255] (grids: [1, 1000]).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from kites_b200 import capi

OPS = {"sssp": capi.OP_SSSP, "bfs": capi.OP_BFS}
STRATEGIES = {"plain": capi.STRATEGY_PLAIN, "auto": capi.STRATEGY_AUTO}
PAGERANK_ITERATIONS = 20
DAMPING = 0.85


def listed():
    return [
        # The drop-in call on a small social graph: the caller's own values
        # and frontier go in from the host, process() runs to the fixed
        # point, the values come back to the host.
        {"name": "process_7k", "kind": "process", "graph": "rmat", "n": 7115, "m": 103689,
         "op": "sssp", "strategy": "plain"},
        # One BFS query on a mid-size graph, default options.
        {"name": "bfs_plain_rmat16", "kind": "single", "graph": "rmat", "n": 60013, "m": 983040,
         "op": "bfs", "strategy": "plain"},
        # Shortest paths on a road-like graph: thousands of thin wavefronts.
        {"name": "sssp_plain_grid512", "kind": "single", "graph": "grid", "n": 512 * 512,
         "m": 4 * 512 * 511, "op": "sssp", "strategy": "plain"},
        # One shortest-path query on a large power-law graph, default options.
        {"name": "sssp_plain_rmat22", "kind": "single", "graph": "rmat", "n": 1 << 22,
         "m": 16 << 22, "op": "sssp", "strategy": "plain"},
        # The same with the learned selector, on a graph of odd size.
        {"name": "sssp_auto_rmat21", "kind": "single", "graph": "rmat", "n": 2000003,
         "m": 31999999, "op": "sssp", "strategy": "auto"},
        # BFS on a uniform random graph through the selector.
        {"name": "bfs_auto_er20", "kind": "single", "graph": "er", "n": 1 << 20, "m": 16 << 20,
         "op": "bfs", "strategy": "auto"},
        # Connected components of a symmetrised graph.
        {"name": "cc_rmat20", "kind": "cc", "graph": "rmat_sym", "n": 1 << 20, "m": 32 << 20,
         "op": "cc", "strategy": "plain"},
        # PageRank, 20 steps.
        {"name": "pagerank_rmat21", "kind": "pagerank", "graph": "rmat", "n": 1 << 21,
         "m": 16 << 21, "op": "pagerank", "strategy": "plain"},
        # A small batch of queries answered together.
        {"name": "batch16_bfs_rmat17", "kind": "batch", "graph": "rmat", "n": 131071,
         "m": 2097143, "op": "bfs", "strategy": "plain", "k": 16},
        # The benchmark's own workload: 64 sources, learned and batched.
        {"name": "batch64_auto_rmat24", "kind": "batch", "graph": "rmat", "n": 1 << 24,
         "m": 16 << 24, "op": "sssp", "strategy": "auto", "k": 64},
        # Many small graphs of uneven size answered in one call.
        {"name": "multi_seed_64", "kind": "multi", "graph": "union", "n": 64 * 12000,
         "m": 64 * 12000 * 16, "parts": 64, "op": "sssp", "strategy": "plain"},
        # A new edge list on the device: build the graph and answer one query.
        {"name": "ingest_rmat20", "kind": "ingest", "graph": "rmat", "n": 1 << 20, "m": 16 << 20,
         "op": "sssp", "strategy": "plain"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["process", "single", "single", "grid", "cc", "pagerank", "batch", "batch",
                       "multi", "ingest"])
    if kind == "grid":
        side = _log_uniform(rng, 64, 640)
        return {"kind": "single", "graph": "grid", "n": side * side, "m": 4 * side * (side - 1),
                "op": rng.choice(["sssp", "bfs"]), "strategy": rng.choice(["plain", "auto"])}
    if kind == "multi":
        parts = _log_uniform(rng, 8, 500)
        n = parts * _log_uniform(rng, 1000, 16000)
        return {"kind": kind, "graph": "union", "n": n, "m": n * rng.randint(4, 24),
                "parts": parts, "op": rng.choice(["sssp", "bfs"]), "strategy": "plain"}
    top = {"process": 300000, "batch": 2000000, "ingest": 4000000}.get(kind, 5000000)
    n = _log_uniform(rng, 2000, top)
    m = n * rng.randint(4, 20) + rng.randint(0, 999)
    graph = rng.choice(["rmat", "rmat", "er"])
    if kind == "cc":
        return {"kind": kind, "graph": graph + "_sym", "n": n, "m": m // 2 * 2, "op": "cc",
                "strategy": "plain"}
    if kind == "pagerank":
        return {"kind": kind, "graph": graph, "n": n, "m": m, "op": "pagerank",
                "strategy": "plain"}
    case = {"kind": kind, "graph": graph, "n": n, "m": m, "op": rng.choice(["sssp", "bfs"]),
            "strategy": "plain" if kind == "process" else rng.choice(["plain", "auto"])}
    if kind == "batch":
        case["k"] = rng.choice([16, 32, 64, 64, 128, 256])
    return case


# ---- inputs -------------------------------------------------------------------

def _rmat(n, m, scale, gen):
    """(src, dst) of m R-MAT edges; n and scale are ints or per-edge tensors."""
    levels = int(scale.max()) if torch.is_tensor(scale) else scale
    src = torch.zeros(m, dtype=torch.int32, device="cuda")
    dst = torch.zeros(m, dtype=torch.int32, device="cuda")
    for level in range(levels):
        r = torch.rand(m, device="cuda", generator=gen)
        down = r >= 0.76                                # quadrants c and d
        right = ((r >= 0.57) & ~down) | (r >= 0.95)     # quadrants b and d
        if torch.is_tensor(scale):
            live = scale > level
            down &= live
            right &= live
            src = torch.where(live, src * 2, src)
            dst = torch.where(live, dst * 2, dst)
        else:
            src *= 2
            dst *= 2
        src += down
        dst += right
    src %= n
    dst %= n
    loops = src == dst
    dst = torch.where(loops, (dst + 1) % n, dst)
    return src, dst


def _edges(case, seed):
    """(src, dst, weights, first vertex of each part) on the GPU, int32."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1 + seed)
    graph, n, m = case["graph"], case["n"], case["m"]
    first = None
    top = 256
    if graph == "grid":
        side = math.isqrt(n)
        ids = torch.arange(n, dtype=torch.int32, device="cuda").view(side, side)
        a = torch.cat([ids[:, :-1].reshape(-1), ids[:-1].reshape(-1)])
        b = torch.cat([ids[:, 1:].reshape(-1), ids[1:].reshape(-1)])
        src, dst = torch.cat([a, b]), torch.cat([b, a])
        top = 1001
    elif graph == "union":
        parts = case["parts"]
        # Part sizes log-uniform over a factor of 100, scaled to n in all.
        x = torch.rand(parts, device="cuda", generator=gen, dtype=torch.float64)
        size = torch.exp(x * math.log(100.0))
        size = torch.clamp((size / size.sum() * n).floor().long(), min=2)
        size[torch.argmax(size)] += n - size.sum()
        first = torch.cumsum(size, 0) - size
        count = torch.clamp((size * (m / n)).floor().long(), min=1)
        count[torch.argmax(size)] += m - count.sum()
        part = torch.repeat_interleave(torch.arange(parts, device="cuda"), count)
        scale = torch.ceil(torch.log2(size.double())).int()
        src, dst = _rmat(size[part].int(), m, scale[part], gen)
        src += first[part].int()
        dst += first[part].int()
    else:
        half = m // 2 if graph.endswith("_sym") else m
        if graph.startswith("rmat"):
            src, dst = _rmat(n, half, max(1, (n - 1).bit_length()), gen)
        else:
            src = torch.randint(0, n, (half,), device="cuda", generator=gen, dtype=torch.int32)
            dst = torch.randint(0, n, (half,), device="cuda", generator=gen, dtype=torch.int32)
        if graph.endswith("_sym"):
            src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    w = torch.randint(1, top, (m,), device="cuda", generator=gen, dtype=torch.int32)
    return src, dst, w, first


def _sources(src, n, count, seed):
    """`count` vertices that have out-edges, uniform among them."""
    has = torch.zeros(n, dtype=torch.bool, device="cuda")
    has[src.long()] = True
    ids = torch.nonzero(has).view(-1).cpu().numpy()
    pick = np.random.default_rng(1000 + seed).integers(0, ids.shape[0], count)
    return ids[pick].astype(np.uint32)


_engine = None


def engine():
    """One engine per process, as a server keeps it."""
    global _engine
    if _engine is None:
        _engine = capi.Engine(0)
    return _engine


def prepare(case, seed):
    eng = engine()
    kind, n = case["kind"], case["n"]
    src, dst, w, first = _edges(case, seed)
    weights = w if case["op"] == "sssp" else None
    state = {"kind": kind, "n": n, "op": OPS.get(case["op"]),
             "opts": capi.default_opts(strategy=STRATEGIES[case["strategy"]])}
    if kind == "multi":
        # One seed per part: a vertex of it that has out-edges.
        part = torch.searchsorted(first, src.long(), right=True) - 1
        seeds = torch.zeros(first.shape[0], dtype=torch.int64, device="cuda")
        seeds.scatter_reduce_(0, part, src.long(), "amax", include_self=False)
        state["seeds"] = seeds.cpu().numpy().astype(np.uint32)
    elif kind in ("single", "process", "ingest"):
        state["source"] = int(_sources(src, n, 1, seed)[0])
    elif kind == "batch":
        state["sources"] = _sources(src, n, case["k"], seed)
    if kind == "process":
        # The example's pre-processing: distance 0 at the source, the
        # source's out-neighbours in the first frontier.
        source = state["source"]
        values = np.full(n, capi.INF, np.uint32)
        values[source] = 0
        bits = np.zeros((n + 31) // 32 * 32, np.uint8)
        bits[dst[src == source].cpu().numpy()] = 1
        state["values"] = values
        state["bits"] = np.packbits(bits, bitorder="little").view(np.uint32)
    elif kind == "batch":
        state["out"] = torch.empty((n, case["k"]), dtype=torch.int32, device="cuda")
    elif kind == "pagerank":
        state["out"] = torch.empty(n, dtype=torch.float32, device="cuda")
    else:
        state["out"] = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    if kind == "ingest":
        state["edges"] = (src, dst, weights)
    else:
        state["graph"] = capi.Graph.from_edges(eng, n, src, dst, weights)
    return state


# ---- the call -----------------------------------------------------------------

def run(state):
    kind, op, opts = state["kind"], state["op"], state["opts"]
    if kind == "ingest":
        src, dst, w = state["edges"]
        g = capi.Graph.from_edges(engine(), state["n"], src, dst, w)
        out, _ = g.sssp(state["source"], op=op, out=state["out"], opts=opts)
        g.close()
        return out
    g = state["graph"]
    if kind == "process":
        g.set_values(state["values"])
        g.set_frontier(state["bits"], state["n"])
        g.process(op, opts=opts)
        return g.get_values(state["n"])
    if kind == "single":
        return g.sssp(state["source"], op=op, out=state["out"], opts=opts)[0]
    if kind == "batch":
        return g.sssp_batch(state["sources"], op=op, out=state["out"], opts=opts)[0]
    if kind == "multi":
        return g.sssp_multi_seed(state["seeds"], op=op, out=state["out"], opts=opts)[0]
    if kind == "cc":
        return g.cc(out=state["out"], opts=opts)[0]
    return g.pagerank(iterations=PAGERANK_ITERATIONS, damping=DAMPING, out=state["out"],
                      opts=opts)[0]


def work(case):
    n, m = case["n"], case["m"]
    weights = 4 if case["op"] == "sssp" else 0
    out = 4 * n * case.get("k", 1)
    if case["kind"] == "ingest":       # the edge list in, the CSC and the distances out
        return {"bytes": (8 + weights) * m + (4 + weights) * m + 4 * n + out, "flops": 0}
    steps = PAGERANK_ITERATIONS if case["kind"] == "pagerank" else 1
    return {"bytes": (4 + weights) * m + 4 * n + out, "flops": 2 * m * steps * case.get("k", 1)}


def exact(case, seed):
    """PageRank in 64 bits; distances and labels are whole numbers."""
    if case["kind"] != "pagerank":
        return None
    n = case["n"]
    src, dst, _, _ = _edges(case, seed)
    src, dst = src.long(), dst.long()
    deg = torch.bincount(src, minlength=n).double()
    inv = torch.where(deg > 0, 1.0 / deg.clamp(min=1), torch.zeros_like(deg))
    pr = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    for _ in range(PAGERANK_ITERATIONS):
        y = torch.zeros_like(pr).index_add_(0, dst, (pr * inv)[src])
        pr = (1.0 - DAMPING) / n + DAMPING * y
    return pr
