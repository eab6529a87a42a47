"""Batched queries in one persistent kernel (wedge_cuda_batch_*): every query's
result equals its own CPU run -- SSSP distances bit-exact, BFS levels exact
with every parent an in-neighbour one level up -- on a small mixed batch, on
the full 256 BFS + 256 SSSP over 64 graphs workload, with and without the
captured CUDA graph, under every tuning the autotuner may pick."""
import os

import numpy as np
import pytest

from helpers import UNREACHED, check_bfs_sorted, levels_from_parents

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 8


@pytest.fixture(scope="module")
def W(engine_lib):
    return engine_lib


@pytest.fixture(scope="module")
def O(oracle_lib):
    return oracle_lib


def _expected(O, params, queries):
    """per query: ('sssp', distances) or ('bfs', levels), from the oracle run alone"""
    want = {}
    for gi, (scale, ef, seed, _h) in enumerate(params):
        mine = [(qi, app, root) for qi, (g, app, root) in enumerate(queries) if g == gi]
        if not mine:
            continue
        V, s, d = O.rmat(scale, ef, seed, threads=THREADS)
        s, d = O.sort_edges(V, s, d, threads=THREADS)
        w = O.weights(s, d)
        gb = O.Graph.from_edges(V, s, d, O.BFS, threads=THREADS)
        gs = O.Graph.from_edges(V, s, d, O.SSSP, w, threads=THREADS)
        for qi, app, root in mine:
            if app == 0:  # BFS
                p, _, _ = gb.run(root=root, threads=THREADS)
                want[qi] = ("bfs", levels_from_parents(p, root), V, s, d, root)
            else:
                want[qi] = ("sssp", gs.run(root=root, threads=THREADS)[0])
        gb.close()
        gs.close()
    return want


def _check(batch, want):
    for qi, exp in want.items():
        got = batch.read_result(qi)
        if exp[0] == "sssp":
            assert np.array_equal(got, exp[1]), f"query {qi}: SSSP distances differ"
        else:
            _, levels, V, s, d, root = exp
            check_bfs_sorted(got, V, s, d, root, levels)


def test_small_mixed_batch(W, O):
    from wedge_gb300 import batch as B

    params = B.graph_params(num_graphs=8, seed=9, scales=(8, 12), edge_factors=(4, 24))
    qs = B.queries(params, 3, 3)
    qs.append((0, W.APP_BFS, 10**9))  # out-of-range root selects vertex 0 (main.c:81-85)
    want = _expected(O, params, [(g, a, r if r < (1 << params[g][0]) else 0) for g, a, r in qs])
    graphs = B.load_graphs(params)
    with W.Batch(graphs, qs) as b:
        st = b.run()
        assert st["rounds"] >= 2 and st["chunks_pulled"] > 0 and st["captured"] == 0
        _check(b, want)
        it1 = b.iterations().copy()
        st2 = b.run(flags=W.FLAG_GRAPH)
        assert st2["captured"] == 1
        _check(b, want)
        b.run(flags=W.FLAG_GRAPH)  # replay of the captured graph
        _check(b, want)
        # BFS depth is a property of the graph; SSSP's iteration count depends on
        # the order of the asynchronous updates, its distances do not
        bfs = np.array([app == W.APP_BFS for _, app, _ in qs])
        assert np.array_equal(b.iterations()[bfs], it1[bfs])
    for g in graphs:
        g.close()


@pytest.mark.parametrize("tuning", [dict(), dict(threshold_pct=5, grab=1, blocks_per_sm=1, split=8),
                                    dict(threshold_pct=60, grab=32, blocks_per_sm=2, split=1024)])
def test_tunings_agree(W, O, tuning):
    from wedge_gb300 import batch as B

    params = B.graph_params(num_graphs=5, seed=11, scales=(9, 13), edge_factors=(8, 16))
    qs = B.queries(params, 2, 2)
    want = _expected(O, params, qs)
    graphs = B.load_graphs(params)
    with W.Batch(graphs, qs) as b:
        b.run(W.BatchTuning(**tuning) if tuning else None)
        _check(b, want)
    for g in graphs:
        g.close()


def test_full_workload_64_graphs(W, O):
    """256 BFS + 256 SSSP over 64 R-MAT graphs, scales 12-20, edge factors 8-32, seed 4"""
    from wedge_gb300 import autotune as A
    from wedge_gb300 import batch as B

    params = B.graph_params()
    qs = B.queries(params)
    assert len(params) == 64 and len(qs) == 512
    assert {p[0] for p in params} <= set(range(12, 21)) and {p[1] for p in params} <= set(range(8, 33))
    graphs = B.load_graphs(params)
    with W.Batch(graphs, qs) as b:
        st = b.run(A.load_tuning(), flags=W.FLAG_GRAPH)
        print("batch of 512 queries:", st)
        want = _expected(O, params, qs)
        _check(b, want)
    for g in graphs:
        g.close()


@pytest.mark.parametrize("chunks", [0, 1])
@pytest.mark.parametrize("own", [1, 127, 128, 129, 700])
def test_batch_of_shards(W, monkeypatch, chunks, own):
    """queries over destination-range shards: a vertex's out-degree is the whole
    graph's, its out-list the shard's part of it (`own` of 40,000 edges here)"""
    from helpers import check_bfs

    monkeypatch.setenv("WEDGE_CSRI_CHUNKS", str(chunks))
    rng = np.random.default_rng(own)
    V = 2000
    # the shard of destinations [0, 1000): 0 and `own` hubs point at them, the rest of their edges goes elsewhere
    hubs = np.arange(1, 6)
    s = np.concatenate([[0] * 5, np.repeat(hubs, own), rng.integers(0, 1000, 3000)])
    d = np.concatenate([hubs, rng.integers(0, 1000, 5 * own), rng.integers(0, 1000, 3000)])
    order = np.lexsort((s, d))
    s, d = s[order].astype(np.uint32), d[order].astype(np.uint32)
    w = rng.integers(1, 256, len(s)).astype(np.uint64)
    outdeg = np.bincount(s, minlength=V).astype(np.uint64)
    outdeg[:6] += 40_000
    fw = (w.astype(np.float64) / 4.0).view(np.uint64)
    with W.Graph.shard(V, s, d, outdeg, len(s) + 240_000, w) as g, \
            W.Graph.shard(V, s, d, outdeg, len(s) + 240_000, fw, W.WEIGHTS_F64) as gf:
        queries = [(i, app, root) for i in (0, 1) for app in (W.APP_SSSP, W.APP_BFS) for root in (0, 1, 500)]
        with W.Batch([g, gf], queries) as b:
            for threshold_pct in (1, 100):
                b.run(W.BatchTuning(threshold_pct=threshold_pct))
                for q, (i, app, root) in enumerate(queries):
                    got = b.read_result(q)
                    if app == W.APP_BFS:
                        check_bfs(got, V, s, d, root)
                        continue
                    dist = np.full(V, np.inf)
                    dist[root] = 0.0
                    wt = fw.view(np.float64) if i else w.astype(np.float64)
                    while True:  # exact: small whole numbers and quarters
                        new = dist.copy()
                        np.minimum.at(new, d, dist[s] + wt)
                        if np.array_equal(new, dist):
                            break
                        dist = new
                    none = np.isinf(dist)
                    expect = dist.view(np.uint64) if i else np.where(none, UNREACHED, np.where(none, 0.0, dist).astype(np.uint64))
                    assert np.array_equal(got, expect), (i, root, threshold_pct)


def test_failed_read_leaves_the_buffer(W):
    """no device memory for the staging of a result: the call says so, and the
    caller's buffer is as it was; with memory again it is read"""
    import ctypes

    import torch

    with W.Graph.rmat(22, 1, 3) as g, W.Batch([g], [(0, W.APP_BFS, 0)]) as b:
        b.run()
        out = np.full(g.V, 0xABABABABABABABAB, np.uint64)
        held = []
        for size in (1 << 30, 1 << 27, 1 << 25):  # the staging takes 32 MB
            try:
                while True:
                    held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                pass
        read = lambda: W.lib().wedge_cuda_batch_read_result(  # noqa: E731
            b._h, 0, out.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(out.nbytes))
        rc = read()
        held.clear()
        torch.cuda.empty_cache()
        assert rc != 0 and np.all(out == 0xABABABABABABABAB)
        assert read() == 0
        g.run(W.APP_BFS)
        assert np.array_equal(out == UNREACHED, g.read_results() == UNREACHED)
