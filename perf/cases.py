"""The work this framework is timed on, one public call path per case.

A case is a dict of plain values.  ``prepare`` makes the graph on the GPU from the seed alone and loads
it, as a program does once; ``run`` is one pass of the application over the loaded graph through the
Python front end (or, where a program hands in its own page-locked buffers, the C ABI the front end
wraps), results read back to host memory.

Graphs: ``rmat`` (R-MAT a=0.57, b=c=0.19, any vertex count: draws outside [0, V) are dropped), ``er``
(uniform pairs), ``grid`` (a road-like 2-D mesh in row-major order with a quarter of the streets missing: low
degree, long diameter).  ``degree`` is the number of directed draws per vertex, before duplicates and
self-loops are removed; CC and ingest graphs hold both directions of every edge.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "grazelle-ppopp18_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

_MASK = 0xFFFFFFFF
_CHUNK = 1 << 26


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # PageRank as on a small web or citation crawl, queried interactively: launches and latency
        {"name": "pr_rmat_4k", "app": "pr", "graph": "rmat", "vertices": 4096, "degree": 16, "iterations": 16, "damping": 0.875},
        # the repository's PageRank configuration: R-MAT 20, 16 iterations, d = 0.85
        {"name": "pr_rmat_1m", "app": "pr", "graph": "rmat", "vertices": 1 << 20, "degree": 16, "iterations": 16, "damping": 0.85},
        # a graph without hubs and with a ragged vertex count
        {"name": "pr_er_3m", "app": "pr", "graph": "er", "vertices": 3000017, "degree": 12, "iterations": 10, "damping": 0.85},
        # a social network of twitter's order: the props are larger than L2
        {"name": "pr_rmat_17m", "app": "pr", "graph": "rmat", "vertices": 1 << 24, "degree": 16, "iterations": 16, "damping": 0.85},
        # the largest: source segments, double props
        {"name": "pr_rmat_67m", "app": "pr", "graph": "rmat", "vertices": 1 << 26, "degree": 16, "iterations": 8, "damping": 0.85},
        # components of a small graph, of the repository's headline graph, and of a road network
        {"name": "cc_rmat_4k", "app": "cc", "graph": "rmat", "vertices": 4096, "degree": 16},
        {"name": "cc_rmat_17m", "app": "cc", "graph": "rmat", "vertices": 1 << 24, "degree": 16},
        # BFS: parents and levels of one search of a middling graph, a road network (a thousand short
        # iterations), and a series of searches under the learned switch, as in the BFS benchmark
        {"name": "bfs_rmat_100k", "app": "bfs", "graph": "rmat", "vertices": 100003, "degree": 16, "roots": 1, "learned": False},
        {"name": "bfs_road_250k", "app": "bfs", "graph": "grid", "vertices": 250999, "degree": 4, "roots": 1, "learned": False},
        {"name": "bfs_rmat_17m", "app": "bfs", "graph": "rmat", "vertices": 1 << 24, "degree": 16, "roots": 8, "learned": True},
        # many graphs at once: personalized PageRank and multi-source BFS, 8 instances of each
        {"name": "batch_8_graphs", "app": "batch", "graph": "mixed", "vertices": 1024, "graphs": 8, "growth": 2.5, "degree": 12, "instances": 8, "iterations": 20, "damping": 0.85},
        # edge list in, labels out: load from page-locked pairs (-push derived) and components
        {"name": "ingest_cc_1m", "app": "ingest", "graph": "rmat", "vertices": 1 << 20, "degree": 16},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    app = rng.choice(["pr", "pr", "pr", "cc", "cc", "bfs", "bfs", "batch", "ingest"])
    if app == "pr":
        return {"app": app, "graph": rng.choice(["rmat", "er"]), "vertices": _log_uniform(rng, 1000, 1 << 24), "degree": rng.randint(4, 20),
                "iterations": rng.randint(4, 20), "damping": rng.choice([0.85, 0.875])}
    if app == "cc":
        kind = rng.choice(["rmat", "rmat", "er", "grid"])
        return {"app": app, "graph": kind, "vertices": _log_uniform(rng, 1000, 200000 if kind == "grid" else 1 << 24),
                "degree": 4 if kind == "grid" else rng.randint(3, 16)}
    if app == "bfs":
        kind = rng.choice(["rmat", "rmat", "er", "grid"])
        return {"app": app, "graph": kind, "vertices": _log_uniform(rng, 1000, 250000 if kind == "grid" else 1 << 24),
                "degree": 4 if kind == "grid" else rng.randint(4, 16), "roots": 1 if kind == "grid" else rng.randint(1, 8),
                "learned": rng.random() < 0.5}
    if app == "batch":
        return {"app": app, "graph": "mixed", "vertices": rng.randint(100, 1500), "graphs": rng.randint(2, 8), "growth": rng.uniform(1.2, 2.5),
                "degree": rng.randint(4, 12), "instances": rng.choice([1, 3, 8, 8]), "iterations": rng.randint(5, 20), "damping": 0.85}
    return {"app": app, "graph": rng.choice(["rmat", "er"]), "vertices": _log_uniform(rng, 20000, 1 << 20), "degree": rng.randint(4, 16)}


# ------------------------------------------------------------------ graphs, on the GPU

def _generator(seed, stream):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + 7919 * stream + 1) & 0x7FFFFFFFFFFFFFFF)
    return g


def _draw_edges(kind, V, degree, gen):
    """Directed draws as (src << 32 | dst), int64 on the GPU, not yet deduplicated."""
    dev = "cuda"
    if kind == "grid":
        cols = math.isqrt(V)
        v = torch.arange(V, device=dev)
        right = v[(v % cols != cols - 1) & (v + 1 < V)]
        down = v[v + cols < V]
        a = torch.cat([right, down])
        b = torch.cat([right + 1, down + cols])
        keep = torch.rand(a.shape[0], device=dev, generator=gen) > 0.25
        a, b = a[keep], b[keep]
        return torch.cat([(a << 32) | b, (b << 32) | a])
    m = V * degree
    parts = []
    for lo in range(0, m, _CHUNK):
        n = min(_CHUNK, m - lo)
        if kind == "er":
            s = torch.randint(0, V, (n,), device=dev, generator=gen)
            d = torch.randint(0, V, (n,), device=dev, generator=gen)
        else:
            s = torch.zeros(n, dtype=torch.int64, device=dev)
            d = torch.zeros(n, dtype=torch.int64, device=dev)
            for _ in range(max(1, (V - 1).bit_length())):
                u = torch.rand(n, device=dev, generator=gen)
                s = (s << 1) | (u >= 0.76)
                d = (d << 1) | (((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
                del u
        k = (s << 32) | d
        parts.append(k[(s < V) & (d < V) & (s != d)])
        del s, d, k
    return torch.cat(parts) if len(parts) != 1 else parts[0]


def _edges(case, seed, stream=0, V=None, kind=None, symmetric=None):
    """(dst << 32 | src) keys in -pull order, duplicates and self-loops removed."""
    V = V or case["vertices"]
    kind = kind or case["graph"]
    k = _draw_edges(kind, V, case["degree"], _generator(seed, stream))
    r = (k >> 32) | ((k & _MASK) << 32)
    if symmetric if symmetric is not None else case["app"] in ("cc", "ingest"):
        r = torch.cat([r, k])
    del k
    return torch.unique(r)


def _pairs(keys):
    """Interleaved (src, dst) pairs of -pull order keys."""
    p = torch.empty((keys.shape[0], 2), dtype=torch.int64, device=keys.device)
    torch.bitwise_and(keys, _MASK, out=p[:, 0])
    p[:, 1] = keys >> 32
    return p


def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True)


def _batch_sizes(case):
    return [int(case["vertices"] * case["growth"] ** g) | 1 for g in range(case["graphs"])]


def _batch_kind(g):
    return "er" if g % 3 == 2 else "rmat"


# ------------------------------------------------------------------ prepare / run

def prepare(case, seed):
    from grazelle.batch import Batch
    from grazelle.engine import Graph
    app, V = case["app"], case["vertices"]
    rng = np.random.RandomState((int(seed) * 2654435761 + 12345) & 0x7FFFFFFF)
    if app == "batch":
        B = Batch(0)
        sizes = _batch_sizes(case)
        for g, n in enumerate(sizes):
            keys = _edges(case, seed, g, n, _batch_kind(g), False)
            B.add_graph(n, _pairs(keys).cpu().numpy().reshape(-1).astype(np.uint64))
        B.build()
        k = case["instances"]
        ids = np.stack([rng.randint(0, n, size=(2, k)) for n in sizes]).astype(np.uint32)
        return {"case": case, "batch": B, "seeds": np.ascontiguousarray(ids[:, 0]), "roots": np.ascontiguousarray(ids[:, 1]),
                "ranks": _pinned((sum(sizes), k), torch.float64), "levels": _pinned((sum(sizes), k), torch.int32)}
    keys = _edges(case, seed)
    E = int(keys.shape[0])
    pairs = _pairs(keys)
    pick = (keys[torch.from_numpy(rng.randint(0, E, size=max(1, case.get("roots", 1)))).cuda()] & _MASK).cpu().tolist()
    del keys
    state = {"case": case, "V": V, "E": E, "out": _pinned((V,), torch.float64)}
    G = state["graph"] = Graph(0)
    if app == "ingest":
        state["pairs"] = torch.empty(pairs.shape, dtype=torch.int64, pin_memory=True).copy_(pairs)
    torch.cuda.synchronize()
    if app == "pr":
        G.load_device_pairs(V, E, pairs.data_ptr())
    elif app != "ingest":
        G.load_pull_derive_push(V, E, pairs.data_ptr())
    if app == "bfs":
        state["roots"] = [int(x) for x in pick]
        if case["learned"]:
            from grazelle import native
            from grazelle import switch
            G.set_policy(native.POLICY_LEARNED, switch.pretrained(0))
    del pairs
    torch.cuda.empty_cache()
    return state


def _read_props(state):
    """The vertex props into the program's own page-locked buffer."""
    import ctypes
    G, out = state["graph"], state["out"]
    G._ck(G.lib.grz_read_props(G.h, ctypes.c_void_p(out.data_ptr()), state["V"]))
    return out


def run(state):
    case = state["case"]
    app = case["app"]
    if app == "batch":
        import ctypes
        from grazelle import native
        B, k = state["batch"], case["instances"]
        st = [native.RunStats(), native.RunStats()]
        ms = ctypes.c_float()
        B._ck(B.lib.grz_batch_run(B.h, state["seeds"].ctypes.data, k, case["iterations"], ctypes.c_double(case["damping"]),
                                  state["roots"].ctypes.data, k, state["ranks"].data_ptr(), state["levels"].data_ptr(),
                                  ctypes.byref(st[0]), ctypes.byref(st[1]), ctypes.byref(ms)))
        return {"ranks": state["ranks"], "levels": state["levels"]}
    G = state["graph"]
    if app == "pr":
        G.pr_init(case["damping"]).pr_iterate(case["iterations"])
        return _read_props(state)
    if app == "cc":
        G.cc_run()
        return _read_props(state)
    if app == "ingest":
        G.load_pull_derive_push(state["V"], state["E"], state["pairs"].data_ptr())
        G.cc_run()
        return _read_props(state)
    if case["roots"] == 1:
        parents, levels = G.bfs(state["roots"][0])
        return {"parents": parents, "levels": levels}
    found = []
    for r in state["roots"]:
        G.bfs_run(r)
        # (reached vertices, reached edges, checksum of the levels), as an int64
        found.append([x - (1 << 64) if x >> 63 else x for x in G.digest()])
    return {"digests": np.array(found, dtype=np.int64), "last_parents": _read_props(state)}


# ------------------------------------------------------------------ the work and the exact results

def _edge_count(case):
    if case["app"] == "batch":
        return sum(_batch_sizes(case)) * case["degree"]
    if case["graph"] == "grid":
        return 4 * case["vertices"]
    return case["vertices"] * case["degree"] * (2 if case["app"] in ("cc", "ingest") else 1)


def work(case):
    """Source IDs (4 bytes per edge), row offsets and the per-vertex values, each read once, and the
    results written once: per iteration for PageRank, per run for CC and BFS."""
    E = _edge_count(case)
    V = sum(_batch_sizes(case)) if case["app"] == "batch" else case["vertices"]
    if case["app"] == "pr":
        it = case["iterations"]
        return {"bytes": it * (4 * E + 4 * V + 28 * V) + 8 * V, "flops": it * (E + 3 * V)}
    if case["app"] == "batch":
        k, it = case["instances"], case["iterations"]
        return {"bytes": it * (4 * E + 4 * V + (16 * k + 12) * V) + 12 * k * V, "flops": it * k * (E + 3 * V)}
    if case["app"] == "ingest":
        return {"bytes": 16 * E + 4 * E + 4 * V + 12 * V, "flops": 0}
    if case["app"] == "cc":
        return {"bytes": 4 * E + 4 * V + 12 * V, "flops": 0}
    return {"bytes": case["roots"] * (4 * E + 4 * V + 16 * V), "flops": 0}


def _exact_pagerank(src, dst, V, iterations, d):
    deg = torch.bincount(src, minlength=V).double()
    div = torch.where(deg == 0, torch.full_like(deg, V), deg)
    p = (1.0 / V) / div
    for _ in range(iterations):
        acc = torch.zeros(V, dtype=torch.float64, device="cuda")
        for lo in range(0, src.shape[0], _CHUNK * 4):
            acc.index_add_(0, dst[lo:lo + _CHUNK * 4], p[src[lo:lo + _CHUNK * 4]])
        p = ((acc + (1.0 - acc.sum()) / V) * d + (1.0 - d) / V) / div
    return p


def _exact_ppr(src, dst, V, seeds, iterations, d):
    deg = torch.bincount(src, minlength=V).double()
    div = torch.where(deg == 0, torch.full_like(deg, V), deg)[:, None]
    k = len(seeds)
    hot = torch.zeros((V, k), dtype=torch.float64, device="cuda")
    hot[torch.as_tensor(np.asarray(seeds, dtype=np.int64), device="cuda"), torch.arange(k, device="cuda")] = 1.0
    rank = hot.clone()
    for _ in range(iterations):
        p = rank / div
        acc = torch.zeros_like(rank).index_add_(0, dst, p[src])
        rank = d * acc + hot * (d * (1.0 - acc.sum(0)) + (1.0 - d))
    return rank


def _exact_components(src, dst, V):
    f = torch.arange(V, device="cuda")
    while True:
        g = f[f]
        h = g[src]
        n = g.clone().scatter_reduce_(0, dst, h, "amin")
        n.scatter_reduce_(0, f[dst], h, "amin")
        del h
        n = n[n]
        if torch.equal(n, f):
            return f.double()
        f = n


def exact(case, seed):
    """PageRank and PPR values, and component labels, by plain torch in 64 bits.  BFS returns vertex
    numbers and counts only: no computed numbers."""
    app = case["app"]
    if app == "bfs":
        return None
    if app == "batch":
        rng = np.random.RandomState((int(seed) * 2654435761 + 12345) & 0x7FFFFFFF)
        sizes, k = _batch_sizes(case), case["instances"]
        ids = np.stack([rng.randint(0, n, size=(2, k)) for n in sizes])
        ranks = []
        for g, n in enumerate(sizes):
            keys = _edges(case, seed, g, n, _batch_kind(g), False)
            ranks.append(_exact_ppr(keys & _MASK, keys >> 32, n, ids[g, 0], case["iterations"], case["damping"]))
        return {"ranks": torch.cat(ranks), "levels": None}
    keys = _edges(case, seed)
    src, dst = keys & _MASK, keys >> 32
    del keys
    if app == "pr":
        return _exact_pagerank(src, dst, case["vertices"], case["iterations"], case["damping"])
    return _exact_components(src, dst, case["vertices"])
