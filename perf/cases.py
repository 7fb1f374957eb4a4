"""The work that programs over this framework have it do, as measured cases.

Every case is one pass through the Python entry points of sstgraph_gb300 on a
device-resident graph: update batches (latency-bound, bulk, fused), loading a
graph, the EdgeMap/VertexMap algorithms, pairwise queries, and the mix of a
dynamic graph that is updated and then queried.  Graphs are RMAT
(a=0.57 b=0.19 c=0.19, the ids folded where the vertex count is no power of
two) or Erdos-Renyi, symmetrised, as the benchmark and the tests build them;
`edges` counts generated undirected edges (about 2 x edges are stored).
"""
import math

import numpy as np
import torch

import sstgraph_gb300 as sst

RMAT = (0.57, 0.19, 0.19)


def listed():
    return [
        # a live graph's smallest updates: 100 new edges in, 100 out
        {"name": "update_100_rmat16", "kind": "update", "graph": "rmat",
         "n": 1 << 16, "edges": 16 << 16, "batch": 100},
        # the benchmark's largest update step on its scale-24 graph
        {"name": "update_1e6_rmat24", "kind": "update", "graph": "rmat",
         "n": 1 << 24, "edges": 8 << 24, "batch": 1000000},
        # a writer's backlog: many batches of uneven sizes (log-normal, every
        # fourth a removal) applied as one call
        {"name": "batched_64_rmat20", "kind": "batched", "graph": "rmat",
         "n": 1 << 20, "edges": 8 << 20, "batches": 64, "median": 10000},
        # loading a graph of odd size from its edge list
        {"name": "load_er_300k", "kind": "load", "graph": "er",
         "n": 300007, "edges": 2400000},
        # one traversal of a small graph: latency
        {"name": "bfs_rmat14", "kind": "bfs", "graph": "rmat",
         "n": 1 << 14, "edges": 8 << 14},
        # one traversal of a large graph: throughput
        {"name": "bfs_rmat23", "kind": "bfs", "graph": "rmat",
         "n": 1 << 23, "edges": 8 << 23},
        # the static-analytics PageRank: 20 iterations
        {"name": "pagerank20_rmat22", "kind": "pagerank", "graph": "rmat",
         "n": 1 << 22, "edges": 8 << 22, "iters": 20},
        # components of a uniform graph, with vertices that have no edge
        {"name": "cc_er_2m", "kind": "cc", "graph": "er",
         "n": 2000003, "edges": 7000000},
        # single-source dependency scores
        {"name": "bc_rmat20", "kind": "bc", "graph": "rmat",
         "n": 1 << 20, "edges": 8 << 20},
        # triangles of a mid-sized skewed graph
        {"name": "tc_rmat18", "kind": "tc", "graph": "rmat",
         "n": 1 << 18, "edges": 8 << 18, "per_vertex": False},
        # membership and common neighbours of pairs, half of them edges
        {"name": "pairs_20k_rmat18", "kind": "pairs", "graph": "rmat",
         "n": 1 << 18, "edges": 8 << 18, "pairs": 20000},
        # a served graph: an update, then the queries of the serving mix on
        # the changed graph (BFS, a 5-iteration PageRank refresh, per-vertex
        # triangle counts)
        {"name": "refresh_rmat18", "kind": "refresh", "graph": "rmat",
         "n": 1 << 18, "edges": 8 << 18, "batch": 1000, "vertices": 1000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["update", "update", "batched", "load", "bfs", "bfs", "pagerank",
                       "cc", "bc", "tc", "pairs", "refresh"])
    top = {"update": 4 << 20, "batched": 1 << 20, "load": 300000, "bfs": 4 << 20,
           "pagerank": 2 << 20, "cc": 2000000, "bc": 1 << 20, "tc": 200000,
           "pairs": 200000, "refresh": 1 << 18}[kind]
    low = {"update": 1 << 14, "batched": 1 << 14}.get(kind, 3000)
    n = _log(rng, low, top)
    graph = rng.choice(["rmat", "rmat", "er"])
    edges = int(n * rng.uniform(4.0, 8.0))
    c = {"kind": kind, "graph": graph, "n": n, "edges": edges}
    if kind == "cc" and graph == "er":
        c["edges"] = int(n * rng.uniform(1.0, 4.0))
    elif kind == "tc":
        c["per_vertex"] = rng.random() < 0.5
    elif kind == "update":
        c["batch"] = _log(rng, 100, min(1000000, edges // 8))
    elif kind == "batched":
        c["batches"] = rng.randint(4, 64)
        c["median"] = _log(rng, 100, 10000)
    elif kind == "pagerank":
        c["iters"] = rng.randint(5, 20)
    elif kind == "pairs":
        c["pairs"] = _log(rng, 100, 20000)
    elif kind == "refresh":
        c["batch"] = _log(rng, 100, 1000)
        c["vertices"] = _log(rng, 10, 1000)
    return c


# ---- inputs, from the seed alone ------------------------------------------
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFFFFFF)
    return g


def _edges(case, count, gen):
    """count directed (u, v) pairs of the case's distribution, (count, 2) int32."""
    n = case["n"]
    if case["graph"] == "er":
        return torch.randint(0, n, (count, 2), generator=gen, device="cuda", dtype=torch.int32)
    a, b, c = RMAT
    uv = torch.zeros((count, 2), dtype=torch.int32, device="cuda")
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(count, generator=gen, device="cuda")
        row = r >= a + b
        col = ((r >= a) & ~row) | (r >= a + b + c)
        uv[:, 0] = uv[:, 0] * 2 + row
        uv[:, 1] = uv[:, 1] * 2 + col
    return uv if n & (n - 1) == 0 else uv.remainder_(n)


def _both(e):
    return torch.cat([e, e.flip(1)]).contiguous()


def _pairs(case, seed):
    return _both(_edges(case, case["edges"], _gen(seed, 1)))


def _graph(case, seed):
    """The case's graph, and its (row, col) pairs as inserted."""
    pairs = _pairs(case, seed)
    torch.cuda.synchronize()
    g = sst.SparseMatrixV(case["n"])
    step = 1 << 25
    for i in range(0, pairs.shape[0], step):
        g.insert_batch(pairs[i:i + step])
    g.sync()
    g.release_scratch()
    return g, pairs


def _new_edges(case, g, pairs, count, gen):
    """(batch, fresh): about 5% of the batch's pairs are in the graph already,
    fresh are those that are not."""
    dup = count // 20
    at = torch.randint(0, pairs.shape[0], (dup,), generator=gen, device="cuda")
    batch = torch.cat([_edges(case, count - dup, gen), pairs[at]]).contiguous()
    return batch, _fresh(g, batch)


def _fresh(g, batch):
    torch.cuda.synchronize()
    has = g.has_batch(batch)
    g.sync()
    keep = (has == 0) & (batch[:, 0] != batch[:, 1])
    return batch[keep].contiguous()


def _sizes(case):
    """The batched form's batch sizes: log-normal (sigma 1.5), the same for
    every seed."""
    k, r = case["batches"], np.random.RandomState(case["batches"])
    s = np.exp(math.log(case["median"]) + 1.5 * r.standard_normal(k))
    return np.maximum(1, np.minimum(s, 20.0 * case["median"])).astype(np.int64)


def _ops(k):
    return [0 if i % 4 == 3 else 1 for i in range(k)]


def _offsets(sizes):
    off = np.zeros(len(sizes) + 1, np.int64)
    off[1:] = np.cumsum(sizes)
    return torch.from_numpy(off).cuda()


def _i32(*shape):
    return torch.empty(shape, dtype=torch.int32, device="cuda")


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    s = {"case": case}
    if kind == "load":
        s["pairs"] = _pairs(case, seed)
        s["degrees"] = _i32(n)
        return s
    g, pairs = _graph(case, seed)
    s["g"] = g
    gen = _gen(seed, 2)
    src = int(pairs[int(torch.randint(0, pairs.shape[0], (1,), generator=gen, device="cuda"))][0])
    if kind == "update":
        s["batch"], s["fresh"] = _new_edges(case, g, pairs, case["batch"], gen)
        s["has"] = torch.empty(case["batch"], dtype=torch.uint8, device="cuda")
        s["degrees"] = _i32(n)
    elif kind == "batched":
        sizes = _sizes(case)
        ops = _ops(len(sizes))
        parts, undo_in, undo_out = [], [], []
        for k, op in zip(sizes, ops):
            if op:
                b, fresh = _new_edges(case, g, pairs, int(k), gen)
                undo_out.append(fresh)
            else:
                b = pairs[torch.randint(0, pairs.shape[0], (int(k),), generator=gen, device="cuda")]
                undo_in.append(b)
            parts.append(b)
        s["seq"] = (torch.cat(parts).contiguous(), _offsets(sizes))
        s["ops"] = ops
        # and back: what went in and was not there before out, then what was
        # there before in again
        back = undo_out + undo_in
        s["back"] = (torch.cat(back).contiguous(), _offsets([len(b) for b in back]))
        s["back_ops"] = [0] * len(undo_out) + [1] * len(undo_in)
        s["has"] = torch.empty(s["seq"][0].shape[0], dtype=torch.uint8, device="cuda")
        s["degrees"] = _i32(n)
    elif kind == "bfs":
        s["src"], s["out"] = src, _i32(n)
    elif kind == "pagerank":
        s["out"] = torch.empty(n, dtype=torch.float64, device="cuda")
    elif kind == "cc":
        s["out"] = _i32(n)
    elif kind == "bc":
        s["src"], s["out"] = src, torch.empty(n, dtype=torch.float64, device="cuda")
    elif kind == "pairs":
        k = case["pairs"]
        at = torch.randint(0, pairs.shape[0], (k // 2,), generator=gen, device="cuda")
        other = torch.randint(0, n, (k - k // 2, 2), generator=gen, device="cuda",
                              dtype=torch.int32)
        s["pairs"] = torch.cat([pairs[at], other]).contiguous()
        s["has"] = torch.empty(k, dtype=torch.uint8, device="cuda")
        # the outputs that the framework allocates come from this stream's pool
        s["stream"] = torch.cuda.Stream()
        g.set_stream(s["stream"].cuda_stream)
    elif kind == "refresh":
        s["batch"] = _both(_edges(case, case["batch"], gen))
        s["fresh"] = _fresh(g, s["batch"])
        s["src"], s["depths"] = src, _i32(n)
        s["ranks"] = torch.empty(n, dtype=torch.float64, device="cuda")
        v = torch.randint(0, n, (case["vertices"],), generator=gen, device="cuda")
        s["vertices"] = v.cpu().numpy().astype(np.uint32)
    torch.cuda.synchronize()
    return s


def run(s):
    case, g = s["case"], s.get("g")
    kind = case["kind"]
    if kind == "update":
        bad = g.insert_batch(s["batch"])
        g.degrees(out=s["degrees"])
        g.remove_batch(s["fresh"])
        g.has_batch(s["batch"], out=s["has"])
        return {"invalid": bad, "edges": g.M(), "degrees": s["degrees"], "has": s["has"]}
    if kind == "batched":
        bad = g.update_batches(s["seq"], s["ops"])
        g.degrees(out=s["degrees"])
        g.has_batch(s["seq"][0], out=s["has"])
        m = g.M()
        g.update_batches(s["back"], s["back_ops"])
        return {"invalid": bad, "edges": [m, g.M()], "degrees": s["degrees"], "has": s["has"]}
    if kind == "load":
        g = sst.SparseMatrixV(case["n"])
        bad = g.insert_batch(s["pairs"])
        g.degrees(out=s["degrees"])
        m = g.M()
        g.close()
        return {"invalid": bad, "edges": m, "degrees": s["degrees"]}
    if kind == "bfs":
        return sst.BFS(g, s["src"], depths=True, out=s["out"])
    if kind == "pagerank":
        return sst.PR_S(g, case["iters"], out=s["out"])
    if kind == "cc":
        return sst.CC(g, out=s["out"])
    if kind == "bc":
        return sst.BC(g, s["src"], out=s["out"])
    if kind == "tc":
        return sst.TC(g, per_vertex=case["per_vertex"])
    if kind == "pairs":
        with torch.cuda.stream(s["stream"]):
            g.has_batch(s["pairs"], out=s["has"])
            return {"has": s["has"], "common": g.common_neighbors_batch(s["pairs"])}
    if kind == "refresh":
        g.insert_batch(s["batch"])
        sst.BFS(g, s["src"], depths=True, out=s["depths"])
        sst.PR_S(g, 5, out=s["ranks"])
        tri = sst.TC_vertices(g, s["vertices"])
        g.remove_batch(s["fresh"])
        return {"depths": s["depths"], "ranks": s["ranks"], "triangles": tri, "edges": g.M()}
    raise ValueError(kind)


def work(case):
    """Bytes: ids of the edges that are read (4 each) and the per-vertex
    inputs and outputs, once; for an update the batch, and one sector of a row
    read and written per edge that changes."""
    kind, n, m = case["kind"], case["n"], 2 * case["edges"]
    flops = 0
    if kind == "update":
        b = 2 * case["batch"] * (8 + 64) + case["batch"] * 9 + 8 * n
    elif kind == "batched":
        k = int(_sizes(case).sum())
        b = 2 * k * (8 + 64) + 9 * k + 8 * n
    elif kind == "load":
        b = 8 * m + 4 * m + 24 * n
    elif kind == "bfs":
        b = 4 * m + 20 * n
    elif kind == "pagerank":
        b, flops = case["iters"] * (4 * m + 24 * n), case["iters"] * 2 * m
    elif kind == "cc":
        b = 4 * m + 20 * n
    elif kind == "bc":
        b, flops = 8 * m + 28 * n, 4 * m
    elif kind == "tc":
        b = 4 * m + 16 * n
    elif kind == "pairs":
        b = case["pairs"] * (8 + 1 + 8 + 2 * (16 + 4 * max(1, m // n)))
    else:
        b = 4 * case["batch"] * (8 + 64) + 4 * m + 20 * n + 5 * (4 * m + 24 * n)
        b += case["vertices"] * 4 * (m // n) * (m // n)
        flops = 5 * 2 * m
    return {"bytes": float(b), "flops": float(flops)}


# ---- the floating outputs, in 64 bits -------------------------------------
def _distinct(n, pairs):
    """(u, v) of the distinct edges without self-loops, u ascending."""
    p = pairs[pairs[:, 0] != pairs[:, 1]]
    k = torch.unique(p[:, 0].long() * n + p[:, 1].long())
    return k // n, k % n


def _pagerank(n, u, v, iters, damping=0.85):
    deg = torch.bincount(u, minlength=n)
    some = deg > 0
    base = (1.0 - damping) / n
    r = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    for _ in range(iters):
        c = torch.where(some, r / deg.clamp(min=1), 0.0)
        t = torch.segment_reduce(c[v], "sum", lengths=deg, initial=0.0)
        r = torch.where(some, base + damping * t, base)
    return r


def _dependencies(n, u, v, src):
    depth = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    sigma = torch.zeros(n, dtype=torch.float64, device="cuda")
    depth[src], sigma[src] = 0, 1.0
    levels = []
    while True:
        d = len(levels)
        near = depth[u] == d
        depth[v[near & (depth[v] < 0)]] = d + 1
        down = near & (depth[v] == d + 1)
        if not bool(down.any()):
            break
        a, b = u[down], v[down]
        sigma.index_add_(0, b, sigma[a])
        levels.append((a, b))
    dep = torch.zeros(n, dtype=torch.float64, device="cuda")
    for a, b in reversed(levels):
        dep.index_add_(0, a, sigma[a] * ((1.0 + dep[b]) / sigma[b]))
    return dep


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind not in ("pagerank", "bc", "refresh"):
        return None  # whole numbers only
    pairs = _pairs(case, seed)
    gen = _gen(seed, 2)
    src = int(pairs[int(torch.randint(0, pairs.shape[0], (1,), generator=gen, device="cuda"))][0])
    if kind == "refresh":
        more = _both(_edges(case, case["batch"], gen))
        u, v = _distinct(n, torch.cat([pairs, more]))
        return {"depths": None, "ranks": _pagerank(n, u, v, 5), "triangles": None, "edges": None}
    u, v = _distinct(n, pairs)
    return _pagerank(n, u, v, case["iters"]) if kind == "pagerank" else _dependencies(n, u, v, src)
