"""The workloads this engine's speed is measured on.

Every case is a call a user's program makes through the package's public entry
points (wedge_gb300.Graph, wedge_gb300.Batch): one traversal or one PageRank of
a graph that stays resident on the GPU, and its results read into page-locked
host memory in the reference's 64-bit representation.  Graphs are the seeded
synthetic ones of the test and benchmark configurations: R-MAT
(0.57/0.19/0.19/0.05, duplicates and self-loops kept) of scales 12 to 26 and
the 4-neighbour grid with 1% random long-range pairs.

`kind` selects the call:
  bfs, cc, sssp   one traversal; `graph` is the device-side loop
                  (FLAG_GRAPH), without it the host drives the iterations as
                  the command line does
  pr              PageRank, `prec` 64 (reference arithmetic) or 32 (compensated)
  batch           SSSP queries over several uneven graphs in one launch
  load            a graph file's image from host memory to the device, one
                  BFS, the results, and the handle closed again: one run of
                  the command line without the disk
"""
from __future__ import annotations

import math

import numpy as np
import torch

import wedge_gb300 as W
from wedge_gb300 import autotune, batch

M64 = (1 << 64) - 1
ABC = (0.57, 0.19, 0.19)
LONG_RANGE = 0.01
DAMPING = 0.85


def listed():
    return [
        # the smallest graph of the batched workload, alone: launches and latency
        {"name": "bfs_rmat12", "kind": "bfs", "scale": 12, "ef": 16, "root": 0, "graph": True},
        # the plain BFS configuration: scale 24, edge factor 16
        {"name": "bfs_rmat24", "kind": "bfs", "scale": 24, "ef": 16, "root": 0, "graph": True},
        # labels of a directed graph as the command line runs them (host-driven loop)
        {"name": "cc_rmat18_directed", "kind": "cc", "scale": 18, "ef": 11, "sym": False, "graph": False},
        # the plain CC configuration: the symmetrised scale-24 graph
        {"name": "cc_rmat24_sym", "kind": "cc", "scale": 24, "ef": 16, "sym": True, "graph": True},
        # the PageRank configuration in the reference's arithmetic: 16 iterations, the graph fits L2
        {"name": "pr64_rmat16", "kind": "pr", "prec": 64, "scale": 16, "ef": 16, "iters": 16, "graph": True},
        # compensated PageRank of an ordinary graph
        {"name": "pr32_rmat20", "kind": "pr", "prec": 32, "scale": 20, "ef": 13, "iters": 20, "graph": True},
        # compensated PageRank of the headline benchmark: 30 iterations over 1.07 G edges
        {"name": "pr32_rmat26", "kind": "pr", "prec": 32, "scale": 26, "ef": 16, "iters": 30, "graph": True},
        # the headline benchmark's SSSP: hash weights 1..255
        {"name": "sssp_rmat26", "kind": "sssp", "on": "rmat", "scale": 26, "ef": 16, "weights": "u64", "root": 0,
         "graph": True},
        # the road-like SSSP configuration: many short iterations
        {"name": "sssp_grid4096", "kind": "sssp", "on": "grid", "side": 4096, "weights": "u64", "root": 0,
         "graph": True},
        # its FP64-weight form on a smaller graph of odd size, host-driven
        {"name": "sssp_grid1001_f64", "kind": "sssp", "on": "grid", "side": 1001, "weights": "f64", "root": 0,
         "graph": False},
        # many queries over graphs of scales 12..20 in one persistent launch
        {"name": "batch_8x4", "kind": "batch", "graphs": 8, "queries": 4, "lo": 12, "hi": 20},
        # a whole run from a file image to results
        {"name": "load_bfs_rmat20", "kind": "load", "scale": 20, "ef": 16, "root": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bfs", "cc", "pr", "pr", "sssp", "sssp", "grid", "batch", "load"])
    graph = rng.random() < 0.7
    ef = rng.randint(8, 32)
    # roots of many and of few out-edges: ids with one set bit
    if kind == "bfs":
        scale = rng.randint(12, 25)
        return {"kind": "bfs", "scale": scale, "ef": ef if scale < 25 else 16, "root": rng.choice([0, 1, 8, 1 << 11]),
                "graph": graph}
    if kind == "cc":
        return {"kind": "cc", "scale": rng.randint(12, 24), "ef": rng.randint(8, 16), "sym": rng.random() < 0.6,
                "graph": graph}
    if kind == "pr":
        prec = rng.choice([32, 64])
        return {"kind": "pr", "prec": prec, "scale": rng.randint(13, 25 if prec == 32 else 23), "ef": rng.randint(8, 16),
                "iters": rng.randint(3, 24), "graph": graph}
    if kind == "sssp":
        scale = rng.randint(12, 25)
        return {"kind": "sssp", "on": "rmat", "scale": scale, "ef": ef if scale < 24 else 14,
                "weights": rng.choice(["u64", "u64", "f64"]), "root": rng.choice([0, 1, 8, 1 << 11]), "graph": graph}
    if kind == "grid":
        return {"kind": "sssp", "on": "grid", "side": _log_int(rng, 65, 3000), "weights": rng.choice(["u64", "f64"]),
                "root": rng.randint(0, 4000), "graph": graph}
    if kind == "batch":
        return {"kind": "batch", "graphs": rng.randint(2, 12), "queries": rng.randint(1, 5), "lo": 12,
                "hi": rng.randint(14, 20)}
    return {"kind": "load", "scale": rng.randint(12, 22), "ef": ef, "root": rng.choice([0, 1, 8])}


# ------------------------------------------------------------------ inputs
def _weight_kind(case):
    return W.WEIGHTS_F64 if case.get("weights") == "f64" else W.WEIGHTS_U64


def _pinned(V):
    return torch.empty(V, dtype=torch.int64, pin_memory=True).numpy().view(np.uint64)


def _batch_graphs(case, seed):
    # the workload's sizes and roots (its seed 4), with edges of this seed
    sizes = batch.graph_params(case["graphs"], 4, (case["lo"], case["hi"]))
    return [(scale, ef, seed * 1000 + i, h) for i, (scale, ef, _s, h) in enumerate(sizes)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        params = _batch_graphs(case, seed)
        graphs = batch.load_graphs(params)
        qs = batch.queries(params, 0, case["queries"])
        return {"kind": kind, "batch": W.Batch(graphs, qs), "n": len(qs), "tuning": autotune.load_tuning()}
    if kind == "load":
        s, d = _rmat_edges(case["scale"], case["ef"], seed, False)
        key = torch.sort((d.to(torch.int64) << 32) | s.to(torch.int64)).values
        V, E = 1 << case["scale"], int(key.numel())
        image = np.empty(2 + 2 * E, np.uint64)
        image[0], image[1] = V, E
        image[2:].reshape(E, 2)[:, 0] = (key & 0xFFFFFFFF).cpu().numpy().view(np.uint64)
        image[2:].reshape(E, 2)[:, 1] = (key >> 32).cpu().numpy().view(np.uint64)
        return {"kind": kind, "image": image.view(np.uint8), "out": _pinned(V),
                "params": W.Params(root=case["root"], flags=W.FLAG_GRAPH)}
    if kind == "sssp" and case["on"] == "grid":
        g = W.Graph.grid(case["side"], LONG_RANGE, seed, _weight_kind(case))
    elif kind == "sssp":
        g = W.Graph.rmat(case["scale"], case["ef"], seed, weight_kind=_weight_kind(case))
    else:
        g = W.Graph.rmat(case["scale"], case["ef"], seed, symmetrise=bool(case.get("sym", False)))
    flags = W.FLAG_GRAPH if case["graph"] else 0
    if kind == "pr":
        app = W.APP_PR
        params = W.Params(num_iterations=case["iters"], damping=DAMPING, flags=flags,
                          precision=W.PREC_FP32C if case["prec"] == 32 else W.PREC_FP64)
    else:
        app = {"bfs": W.APP_BFS, "cc": W.APP_CC, "sssp": W.APP_SSSP}[kind]
        params = W.Params(root=case.get("root", 0), flags=flags)
    # the launch knobs a program takes from the tuning table, where it has the graph's size
    if case.get("on") != "grid":
        name = {"bfs": "bfs", "cc": "cc", "pr": "pr", "sssp": "sssp"}[kind]
        if kind != "pr" or case["prec"] == 32:
            autotune.apply_engine_tuning(g, name, case["scale"], case["ef"])
    real = kind in ("cc", "pr") or case.get("weights") == "f64"
    return {"kind": kind, "g": g, "app": app, "params": params, "out": _pinned(g.V), "real": real}


# -------------------------------------------------------------------- runs
def run(state):
    if state["kind"] == "batch":
        b = state["batch"]
        b.run(state["tuning"], flags=W.FLAG_GRAPH)
        return [b.read_result(i).view(np.int64) for i in range(state["n"])]
    if state["kind"] == "load":
        with W.Graph.load_image(state["image"], W.APP_BFS) as g:
            g.run(W.APP_BFS, state["params"])
            return g.read_results(state["out"]).view(np.int64)
    g = state["g"]
    g.run(state["app"], state["params"])
    return g.read_results(state["out"]).view(np.float64 if state["real"] else np.int64)


def _size(case):
    """(vertices, edges) of a case's graph"""
    if case.get("on") == "grid":
        base = 4 * case["side"] * (case["side"] - 1)
        return case["side"] ** 2, base + int(LONG_RANGE * base)
    E = case["ef"] << case["scale"]
    return 1 << case["scale"], 2 * E if case.get("sym") else E


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = 0
        for scale, ef, _s, _h in _batch_graphs(case, 1):
            b += case["queries"] * ((ef << scale) * 5 + (16 << scale))
        return {"bytes": b, "flops": 0}
    V, E = _size(case)
    if kind in ("bfs", "cc"):
        # one in-edge source of every vertex, its offsets, its result
        return {"bytes": 20 * V, "flops": 0}
    if kind == "load":
        return {"bytes": 16 * E + 4 * E + 20 * V, "flops": 0}
    if kind == "sssp":
        # every source and weight once, offsets, results
        return {"bytes": (12 if case["weights"] == "f64" else 5) * E + 16 * V, "flops": E}
    # sources once an iteration, offsets, ranks read and written, 1/outdegree; the results
    word = 4 if case["prec"] == 32 else 8
    return {"bytes": case["iters"] * (4 * E + (8 + 3 * word) * V) + 8 * V, "flops": case["iters"] * E}


# ------------------------------------------------------------ plain results
def _i64(x):
    return x - (1 << 64) if x >= 1 << 63 else x


def _shr(z, n):
    return (z >> n) & ((1 << (64 - n)) - 1)


def _mix(z):
    z = z + _i64(0x9E3779B97F4A7C15)
    z = (z ^ _shr(z, 30)) * _i64(0xBF58476D1CE4E5B9)
    z = (z ^ _shr(z, 27)) * _i64(0x94D049BB133111EB)
    return z ^ _shr(z, 31)


def _mix_int(z):
    z = (z + 0x9E3779B97F4A7C15) & M64
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
    return z ^ (z >> 31)


CHUNK = 1 << 26


def _rmat_edges(scale, ef, seed, sym):
    """the generator's edges, unsorted, as int32 tensors on the GPU"""
    E = ef << scale
    ta, tab, tabc = (int(x * 4294967296.0) for x in (ABC[0], ABC[0] + ABC[1], ABC[0] + ABC[1] + ABC[2]))
    src = torch.empty(2 * E if sym else E, dtype=torch.int32, device="cuda")
    dst = torch.empty_like(src)
    base = _i64(_mix_int(seed))
    for e0 in range(0, E, CHUNK):
        n = min(CHUNK, E - e0)
        item = torch.arange(e0, e0 + n, device="cuda") << 4
        s = torch.zeros(n, dtype=torch.int64, device="cuda")
        d = torch.zeros_like(s)
        h = None
        for level in range(scale):
            if level % 2 == 0:
                h = _mix(base + (item | (level // 2)))
            u = _shr(h, 32) if level % 2 else h & 0xFFFFFFFF
            bit = 1 << (scale - 1 - level)
            s += (u >= tab) * bit
            d += (((u >= ta) & (u < tab)) | (u >= tabc)) * bit
        src[e0:e0 + n], dst[e0:e0 + n] = s, d
    if sym:
        src[E:], dst[E:] = dst[:E], src[:E]
    return src, dst


def _grid_edges(side, seed):
    V = side * side
    v = torch.arange(V, device="cuda").reshape(side, side)
    pairs = [(v[:, :-1], v[:, 1:]), (v[:-1], v[1:])]
    s = [x.reshape(-1) for a, b in pairs for x in (a, b)]
    d = [x.reshape(-1) for a, b in pairs for x in (b, a)]
    lr = int(LONG_RANGE * float(4 * side * (side - 1)))
    j = torch.arange(lr, device="cuda") << 4
    base = _i64(_mix_int(seed))

    def pick(word):
        h = _mix(base + (j | word))
        return (_shr(h, 32) * V + (((h & 0xFFFFFFFF) * V) >> 32)) >> 32

    return torch.cat(s + [pick(0)]).to(torch.int32), torch.cat(d + [pick(1)]).to(torch.int32)


def _weights(s, d, f64):
    h = ((s.to(torch.int64) << 32) | d.to(torch.int64)) * _i64(0x9E3779B97F4A7C15)
    hi = _shr(h, 32)
    if f64:
        return (hi.to(torch.float64) * 4294967296.0 + (h & 0xFFFFFFFF).to(torch.float64)) * 2.0 ** -64
    return 1 + ((hi * 255) >> 32)


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("cc", "pr", "sssp"):
        return None  # parents: any in-neighbour one level up would do; batch: whole numbers
    if case.get("on") == "grid":
        src, dst = _grid_edges(case["side"], seed)
    else:
        src, dst = _rmat_edges(case["scale"], case["ef"], seed, bool(case.get("sym", False)))
    V, E = _size(case)
    parts = [(src[i:i + CHUNK].long(), dst[i:i + CHUNK].long()) if E <= 4 * CHUNK else (i, min(E, i + CHUNK))
             for i in range(0, E, CHUNK)]

    def edges():
        for a, b in parts:
            yield (src[a:b].long(), dst[a:b].long()) if isinstance(a, int) else (a, b)

    if kind == "pr":
        deg = torch.zeros(V, dtype=torch.float64, device="cuda")
        for s, _ in edges():
            deg += torch.bincount(s, minlength=V).double()
        deg[deg == 0] = float(V)
        rank = (1.0 / V) / deg
        for _ in range(case["iters"]):
            acc = torch.zeros(V, dtype=torch.float64, device="cuda")
            for s, d in edges():
                acc.index_add_(0, d, rank[s])
            rank = ((acc + (1.0 - acc.sum()) / V) * DAMPING + (1.0 - DAMPING) / V) / deg
        return rank
    if kind == "cc":
        x = torch.arange(V, dtype=torch.int64, device="cuda")
        while True:
            y = x.clone()
            for s, d in edges():
                y.scatter_reduce_(0, d, y[s], "amin")
            if torch.equal(x, y):
                return x.double()
            x = y
    f64 = case["weights"] == "f64"
    far = math.inf if f64 else 1 << 62
    x = torch.full((V,), far, dtype=torch.float64 if f64 else torch.int64, device="cuda")
    x[case["root"] if case["root"] < V else 0] = 0
    while True:
        y = x.clone()
        for s, d in edges():
            y.scatter_reduce_(0, d, y[s] + _weights(s, d, f64), "amin")
        if torch.equal(x, y):
            break
        x = y
    return x if f64 else torch.where(x >= far, torch.full_like(x, -1), x)
