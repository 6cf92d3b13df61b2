"""Timed workloads of the framework, through medusa_b200.api.

A case is one call (or a short sequence of calls) that a program using the
library makes, on seeded synthetic graphs of the families the configurations
and tests use: R-MAT with the mild (0.45, 0.15, 0.15) and the skewed
(0.57, 0.19, 0.19) quadrants, uniform random edges, and the road-like grid
with dropped edges and random shortcuts.

listed() -- the named cases; draw(rng) -- one more case of the same ranges;
prepare(case, seed) -- graph handle, sources and output buffers;
run(state) -- one pass; work(case) -- the bytes and operations it needs;
exact(case, seed) -- the same outputs from plain torch in 64 bits.
"""
import math

import numpy as np
import torch

from medusa_b200 import api

DEV = "cuda"
CHUNK = 1 << 26  # edges generated at a time

_contexts = {}


def _context(order="reference"):
    """One context per PageRank order, kept for the life of the program."""
    if order not in _contexts:
        ctx = api.Context(0)
        ctx.set_pagerank_order(api.MB_PR_ORDER_FIXED if order == "fixed" else api.MB_PR_ORDER_REFERENCE)
        _contexts[order] = ctx
    return _contexts[order]


# ---- the cases ------------------------------------------------------------------

def listed():
    return [
        # an interactive query on a small graph: the call's own cost; the
        # levels come back as a host array, the binding's default
        {"name": "bfs-tiny", "kind": "bfs", "graph": "rmat", "V": 1024, "E": 8192, "skew": "mild",
         "out": "host"},
        # a road-like network: high diameter, thousands of small frontiers
        {"name": "bfs-grid-1448", "kind": "bfs", "graph": "grid", "V": 1448 * 1448, "rows": 1448, "out": "device"},
        # the largest graph of the configurations, skewed: few, huge frontiers
        {"name": "bfs-rmat-2e24", "kind": "bfs", "graph": "rmat", "V": 1 << 24, "E": 1 << 28, "skew": "heavy",
         "out": "device"},
        # the benchmark's SSSP: weights 1..1000 on the mild R-MAT
        {"name": "sssp-rmat-2e20", "kind": "sssp", "graph": "rmat", "V": 1 << 20, "E": 1 << 24, "skew": "mild",
         "wmax": 1000, "out": "device"},
        # route lengths on the road-like network, weights 1..100
        {"name": "sssp-grid-1448", "kind": "sssp", "graph": "grid", "V": 1448 * 1448, "rows": 1448, "wmax": 100,
         "out": "device"},
        # ten supersteps on a uniform graph that fits in L2, the default order
        {"name": "pagerank-uniform-2e18", "kind": "pagerank", "graph": "uniform", "V": 1 << 18, "E": 1 << 22,
         "iters": 10, "order": "reference", "out": "device"},
        # twenty supersteps on the largest graph, the default order
        {"name": "pagerank-rmat-2e24", "kind": "pagerank", "graph": "rmat", "V": 1 << 24, "E": 1 << 28,
         "skew": "heavy", "iters": 20, "order": "reference", "out": "device"},
        # the other summation order, on a graph of no round size
        {"name": "pagerank-fixed-ragged", "kind": "pagerank", "graph": "rmat", "V": 1300021, "E": 17000023,
         "skew": "heavy", "iters": 10, "order": "fixed", "out": "device"},
        # many queries at once: 64 BFS sources in one call
        {"name": "bfs64-rmat-2e22", "kind": "bfs", "graph": "rmat", "V": 1 << 22, "E": 1 << 26, "skew": "mild",
         "nsrc": 64, "out": "device"},
        # many queries at once: 32 SSSP sources in one call
        {"name": "sssp32-rmat-2e20", "kind": "sssp", "graph": "rmat", "V": 1 << 20, "E": 1 << 24, "skew": "mild",
         "wmax": 1000, "nsrc": 32, "out": "device"},
        # 64 graphs of 2^10 to 2^16 vertices in one launch: PageRank and one BFS each
        {"name": "many-graphs-64", "kind": "many", "ngraphs": 64, "smin": 10, "smax": 16, "iters": 20},
        # a new weighted edge list: build the graph and answer one SSSP on it
        {"name": "load-sssp-2e20", "kind": "load", "graph": "rmat", "V": 1 << 20, "E": 1 << 24, "skew": "heavy",
         "wmax": 1000, "out": "device"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bfs", "bfs", "sssp", "sssp", "pagerank", "pagerank", "bfs_many", "sssp_many", "many",
                       "load"])
    if kind == "many":
        smax = rng.randint(11, 16)
        return {"kind": "many", "ngraphs": rng.randint(2, 64), "smin": rng.randint(8, 10), "smax": smax,
                "iters": rng.randint(1, 20)}
    hi = {"bfs": 1 << 24, "sssp": 1 << 23, "pagerank": 1 << 23, "bfs_many": 1 << 21, "sssp_many": 1 << 20,
          "load": 1 << 21}[kind]
    V = _log_uniform(rng, 1000, hi)
    graph = rng.choice(["rmat", "rmat", "uniform", "grid"]) if kind != "pagerank" else rng.choice(["rmat", "uniform"])
    c = {"kind": kind.replace("_many", ""), "graph": graph, "out": rng.choice(["device", "device", "host"])}
    if graph == "grid":
        rows = max(4, int(math.sqrt(min(V, 1 << 21)) * rng.uniform(0.5, 1.5)))
        c["rows"] = rows
        c["V"] = rows * max(4, min(V, 1 << 21) // rows)
    else:
        c["V"] = V
        c["E"] = int(V * rng.uniform(4, 20)) | 1
        if graph == "rmat":
            c["skew"] = rng.choice(["mild", "heavy"])
    if kind in ("sssp", "sssp_many", "load"):
        c["wmax"] = rng.choice([100, 1000])
    if kind == "pagerank":
        c["iters"] = rng.randint(1, 20)
        c["order"] = rng.choice(["reference", "reference", "fixed"])
    if kind == "bfs_many":
        c["nsrc"] = rng.randint(2, 64)
    if kind == "sssp_many":
        c["nsrc"] = rng.randint(2, 32)
    return c


# ---- inputs ---------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rmat_edges(gen, V, E, skew):
    a, b, c = (0.57, 0.19, 0.19) if skew == "heavy" else (0.45, 0.15, 0.15)
    scale = max(1, (V - 1).bit_length())
    src = torch.empty(E, dtype=torch.int32, device=DEV)
    dst = torch.empty(E, dtype=torch.int32, device=DEV)
    for e0 in range(0, E, CHUNK):
        n = min(CHUNK, E - e0)
        u = torch.zeros(n, dtype=torch.int32, device=DEV)
        v = torch.zeros(n, dtype=torch.int32, device=DEV)
        for _ in range(scale):
            r = torch.rand(n, device=DEV, generator=gen)
            down = r >= a + b
            right = ((r >= a) & ~down) | (r >= a + b + c)
            u.mul_(2).add_(down)
            v.mul_(2).add_(right)
        if V != 1 << scale:  # no power of two: the ids squeezed into [0, V)
            u = torch.div(u.long() * V, 1 << scale, rounding_mode="floor")
            v = torch.div(v.long() * V, 1 << scale, rounding_mode="floor")
        src[e0:e0 + n] = u
        dst[e0:e0 + n] = v
    return src, dst


def _grid_edges(gen, V, rows):
    """Both directions of every lattice edge but a tenth, plus V / 200 shortcuts."""
    cols = V // rows
    ids = torch.arange(rows * cols, dtype=torch.int32, device=DEV).view(rows, cols)
    u = torch.cat([ids[:, :-1].reshape(-1), ids[:-1].reshape(-1)])
    v = torch.cat([ids[:, 1:].reshape(-1), ids[1:].reshape(-1)])
    keep = torch.rand(u.numel(), device=DEV, generator=gen) >= 0.1
    ends = torch.randint(0, rows * cols, (2, max(1, V // 200)), dtype=torch.int32, device=DEV, generator=gen)
    u, v = torch.cat([u[keep], ends[0]]), torch.cat([v[keep], ends[1]])
    return torch.stack([u, v], 1).reshape(-1), torch.stack([v, u], 1).reshape(-1)


def _edges(case, gen):
    """(src, dst, weights or None), int32 and float32 on the GPU."""
    V = case["V"]
    if case["graph"] == "rmat":
        src, dst = _rmat_edges(gen, V, case["E"], case["skew"])
    elif case["graph"] == "uniform":
        src = torch.randint(0, V, (case["E"],), dtype=torch.int32, device=DEV, generator=gen)
        dst = torch.randint(0, V, (case["E"],), dtype=torch.int32, device=DEV, generator=gen)
    else:
        src, dst = _grid_edges(gen, V, case["rows"])
    w = None
    if case.get("wmax"):
        n = src.numel()
        if case["graph"] == "grid":  # one weight per road, both ways
            w = torch.randint(1, case["wmax"] + 1, (n // 2,), device=DEV, generator=gen).repeat_interleave(2).float()
        else:
            w = torch.empty(n, dtype=torch.float32, device=DEV)
            for e0 in range(0, n, CHUNK):
                k = min(CHUNK, n - e0)
                w[e0:e0 + k] = torch.randint(1, case["wmax"] + 1, (k,), device=DEV, generator=gen)
    return src, dst, w


def _sources(case, gen, src):
    """Distinct vertices with out-edges, uniform among the vertices."""
    V, n = case["V"], case.get("nsrc", 1)
    has = torch.zeros(V, dtype=torch.bool, device=DEV)
    for e0 in range(0, src.numel(), CHUNK):
        has[src[e0:e0 + CHUNK].long()] = True
    order = torch.randperm(V, device=DEV, generator=gen)
    first = order[has[order]][:n]
    if first.numel() < n:
        first = torch.cat([first, order[:n - first.numel()]])
    return first.int().cpu().numpy()


def _inputs(case, seed):
    gen = _generator(seed)
    src, dst, w = _edges(case, gen)
    sources = _sources(case, gen, src) if case["kind"] != "pagerank" else None
    return src, dst, w, sources


def _many_inputs(case, seed):
    """[(V, src, dst)] host arrays with ids local to each graph, and a source per graph."""
    gen = _generator(seed)
    sizes = np.random.default_rng(case["ngraphs"])  # the sizes are the case's, the edges the seed's
    graphs, sources = [], []
    for _ in range(case["ngraphs"]):
        V = 1 << int(sizes.integers(case["smin"], case["smax"] + 1))
        E = int(round(V * float(sizes.uniform(4, 32))))
        src, dst = _rmat_edges(gen, V, E, "mild")
        graphs.append((V, src.cpu().numpy(), dst.cpu().numpy()))
        sources.append(int(graphs[-1][1][0]))
    return graphs, np.array(sources, np.int32)


# ---- one pass -------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "many":
        graphs, sources = _many_inputs(case, seed)
        batch = _context().batch_upload(graphs)
        return {"case": case, "batch": batch, "sources": sources,
                "ranks": torch.empty(batch.total_V, dtype=torch.float32, device=DEV),
                "levels": torch.empty(batch.total_V, dtype=torch.int32, device=DEV)}
    src, dst, w, sources = _inputs(case, seed)
    torch.cuda.synchronize()  # the library reads the edges on its own stream
    state = {"case": case, "sources": sources, "ctx": _context(case.get("order", "reference")), "out": None}
    V, n = case["V"], case.get("nsrc", 1)
    if case["out"] == "device":
        if kind == "pagerank":
            state["out"] = torch.empty(V, dtype=torch.float32, device=DEV)
        else:
            state["out"] = torch.empty((n, V), dtype=torch.int32 if kind == "bfs" else torch.float32, device=DEV)
    if kind == "load":
        state["edges"] = (src, dst, w)
    else:
        state["graph"] = state["ctx"].graph_from_edges(V, src, dst, w)
    return state


def _counts(stats):
    return stats["edges_traversed"], stats["vertices_reached"]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "many":
        ranks, levels, _ = state["batch"].run(case["iters"], state["sources"], state["ranks"], state["levels"])
        return ranks, levels
    if kind == "bfs":
        levels, stats = state["graph"].bfs(state["sources"], out=state["out"])
        return levels, _counts(stats)
    if kind == "sssp":
        dist, stats = state["graph"].sssp(state["sources"], out=state["out"])
        return dist, _counts(stats)
    if kind == "pagerank":
        return state["graph"].pagerank(case["iters"], out=state["out"])[0]
    src, dst, w = state["edges"]
    graph = state["ctx"].graph_from_edges(case["V"], src, dst, w)
    dist, stats = graph.sssp(state["sources"], out=state["out"])
    graph.close()
    return dist, _counts(stats)


# ---- what a pass cannot do without ------------------------------------------------

def _sizes(case):
    if case["kind"] == "many":
        V = case["ngraphs"] * ((1 << (case["smax"] + 1)) - (1 << case["smin"])) / (case["smax"] - case["smin"] + 1)
        return V, 18 * V
    V = case["V"]
    return V, case.get("E", 3.61 * V)  # grid: 2 * 2 * 0.9 lattice edges and 2 / 200 shortcuts per vertex


def work(case):
    """Each graph array read once, each output written once; one operation per
    edge (per source, or per superstep) counts as a flop."""
    V, E = _sizes(case)
    kind, n, iters = case["kind"], case.get("nsrc", 1), case.get("iters", 1)
    if kind == "many":
        # the arrays of each superstep: sources of the in-edges, offsets, contributions in and out
        return {"bytes": iters * (4 * E + 12 * V) + 4 * E + 8 * V, "flops": iters * E}
    if kind == "pagerank":
        return {"bytes": iters * (4 * E + 12 * V) + 4 * V, "flops": iters * E}
    if kind == "bfs":
        return {"bytes": 4 * E + 4 * V + 4 * n * V, "flops": n * E}
    if kind == "sssp":
        return {"bytes": 8 * E + 4 * V + 4 * n * V, "flops": n * E}
    # edges in; offsets, columns, weights of both directions and the message slots out; one SSSP
    return {"bytes": 12 * E + 24 * E + 8 * V + 8 * E + 8 * V, "flops": E}


# ---- the same outputs in 64 bits --------------------------------------------------

def _by_destination(V, src, dst, w):
    """The edges grouped by destination: (sources, weights in 64 bits, group sizes)."""
    order = torch.sort(dst).indices
    src = src[order]
    w = None if w is None else w[order].double()
    del order
    sizes = torch.zeros(V, dtype=torch.int64, device=DEV)
    for e0 in range(0, dst.numel(), CHUNK):
        d = dst[e0:e0 + CHUNK].long()
        sizes.index_add_(0, d, torch.ones_like(d))
    return src, w, sizes


def _shortest(V, grouped, starts):
    """64-bit distances (unit weights without w) from all of `starts` at once; inf: unreached."""
    src, w, sizes = grouped
    dist = torch.full((V,), math.inf, dtype=torch.float64, device=DEV)
    dist[torch.as_tensor(starts, device=DEV).long()] = 0.0
    if src.numel() == 0:
        return dist
    while True:
        msg = dist[src]
        msg += 1.0 if w is None else w
        best = torch.segment_reduce(msg, "min", lengths=sizes, unsafe=True, initial=math.inf)
        del msg
        new = torch.minimum(dist, best)
        if torch.equal(new, dist):
            return dist
        dist = new


def _ranks(V, src, dst, iters, init):
    out = torch.zeros(V, dtype=torch.float64, device=DEV)
    for e0 in range(0, src.numel(), CHUNK):
        s = src[e0:e0 + CHUNK].long()
        out.index_add_(0, s, torch.ones(s.numel(), dtype=torch.float64, device=DEV))
    src, _, sizes = _by_destination(V, src, dst, None)
    rank = init.double().clone()
    for _ in range(iters):
        contrib = torch.where(out > 0, rank / out.clamp(min=1), torch.zeros_like(rank))
        rank = 0.15 + 0.85 * torch.segment_reduce(contrib[src], "sum", lengths=sizes, unsafe=True, initial=0.0)
    return rank


def _levels(dist):
    return torch.where(torch.isinf(dist), torch.full_like(dist, -1.0), dist).to(torch.int32)


def exact(case, seed):
    kind = case["kind"]
    if kind == "many":
        graphs, sources = _many_inputs(case, seed)
        base = np.concatenate([[0], np.cumsum([V for V, _, _ in graphs])])
        V = int(base[-1])
        src = torch.from_numpy(np.concatenate([s + b for (_, s, _), b in zip(graphs, base)]).astype(np.int32)).to(DEV)
        dst = torch.from_numpy(np.concatenate([d + b for (_, _, d), b in zip(graphs, base)]).astype(np.int32)).to(DEV)
        init = torch.cat([torch.full((n,), 1.0 / n, dtype=torch.float64, device=DEV) for n, _, _ in graphs])
        ranks = _ranks(V, src, dst, case["iters"], init)
        return ranks, _levels(_shortest(V, _by_destination(V, src, dst, None), sources + base[:-1]))
    V = case["V"]
    src, dst, w, sources = _inputs(case, seed)
    if kind == "pagerank":
        return _ranks(V, src, dst, case["iters"], torch.full((V,), 1.0 / V, dtype=torch.float64, device=DEV))
    degree = torch.zeros(V, dtype=torch.int64, device=DEV)
    for e0 in range(0, src.numel(), CHUNK):
        s = src[e0:e0 + CHUNK].long()
        degree.index_add_(0, s, torch.ones_like(s))
    grouped = _by_destination(V, src, dst, w)
    del src, dst, w
    rows, edges, reached = [], 0, 0
    for s in sources:
        dist = _shortest(V, grouped, [int(s)])
        hit = ~torch.isinf(dist)
        edges += int(degree[hit].sum())
        reached += int(hit.sum())
        # unreached vertices keep the reference's MEDUSA_MAX
        rows.append(_levels(dist) if kind == "bfs" else torch.where(hit, dist, torch.full_like(dist, 1e9)))
    return torch.stack(rows), (edges, reached)
