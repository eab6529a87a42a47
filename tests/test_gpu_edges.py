"""Small graphs at the sizes where the engine's kernels change course (windows,
pieces, tiles), against plain arithmetic on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bellman_ford(V, src, dst, w, root):
    """least path sums in exact integers; UINT64_MAX = unreached"""
    far = 1 << 62
    dist = np.full(V, far, np.int64)
    dist[root] = 0
    while True:
        new = dist.copy()
        reached = dist[src] < far
        np.minimum.at(new, dst[reached], dist[src[reached]] + w[reached].astype(np.int64))
        if np.array_equal(new, dist):
            return np.where(dist >= far, np.uint64(0xFFFFFFFFFFFFFFFF), dist.astype(np.uint64))
        dist = new


def fans(n, weights, seed):
    """root 0 -> n middle vertices -> three targets; the middle vertices' distances
    are random, the targets' in-edges have `weights`: all in-edges of a target are
    read, some, or one, by how the two compare"""
    rng = np.random.default_rng(seed)
    mid = np.arange(1, n + 1)
    w0 = rng.integers(0, 256, n)
    parts_s, parts_d, parts_w = [np.zeros(n, np.int64)], [mid], [w0]
    for t in range(3):
        parts_s.append(mid)
        parts_d.append(np.full(n, n + 1 + t))
        parts_w.append({"equal": np.full(n, 200), "zero": np.zeros(n, np.int64), "random": rng.integers(0, 256, n),
                        "falling": 255 - (np.arange(n) % 256)}[weights])
    s, d, w = (np.concatenate(x) for x in (parts_s, parts_d, parts_w))
    order = np.lexsort((s, d))
    return n + 4, s[order].astype(np.uint32), d[order].astype(np.uint32), w[order].astype(np.uint64)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 29, 32, 33, 36, 37, 4095, 4128, 4129, 4160, 8300])
@pytest.mark.parametrize("weights", ["equal", "zero", "random", "falling"])
def test_weight_ordered_pull(engine_lib, n, weights):
    """destinations around the in-edge window of a lane (32) and the pieces past it
    (4096), dense and source-filtered, and with a 32-bit limit that some sums pass"""
    W = engine_lib
    V, s, d, w = fans(n, weights, n)
    expect = bellman_ford(V, s, d, w, 0)
    with W.Graph.from_edges(V, s, d, w) as g:
        for limit in (None, 150):
            g.set_knob("sssp_narrow", limit)
            for sched in (W.SCHED_DENSE, W.SCHED_FILTERED, W.SCHED_PLAIN):
                g.run(W.APP_SSSP, W.Params(sched=sched, flags=W.FLAG_GRAPH))
                assert np.array_equal(g.read_results(), expect), (limit, sched)


def fan_in_out(n, seed):
    """0 -> n vertices -> n + 1 -> n vertices again, each with a few random edges:
    out-lists of n destinations, and vertices of one"""
    rng = np.random.default_rng(seed)
    V = 2 * n + 3
    first, hub, second = np.arange(1, n + 1), n + 1, np.arange(n + 2, 2 * n + 2)
    s = [np.zeros(n, np.int64), first, np.full(n, hub), rng.integers(0, V - 1, 2 * n)]
    d = [first, np.full(n, hub), second, rng.integers(0, V - 1, 2 * n)]
    s, d = np.concatenate(s), np.concatenate(d)
    order = np.lexsort((s, d))
    s, d = s[order].astype(np.uint32), d[order].astype(np.uint32)
    return V, s, d, rng.integers(0, 256, len(s)).astype(np.uint64)


def least_labels(V, src, dst):
    x = np.arange(V)
    while True:
        y = x.copy()
        np.minimum.at(y, dst, x[src])
        if np.array_equal(x, y):
            return x.astype(np.float64)
        x = y


def check_traversals(W, V, s, d, w, scheds, flags_list):
    import helpers

    levels = helpers.bfs_levels(V, s, d, 0)
    labels = least_labels(V, s.astype(np.int64), d.astype(np.int64))
    dist = bellman_ford(V, s, d, w, 0)
    fw = (w.astype(np.float64) + 0.25).view(np.uint64)
    with W.Graph.from_edges(V, s, d, w) as g, W.Graph.from_edges(V, s, d, fw, W.WEIGHTS_F64) as gf:
        fdist = None
        parents = None
        for sched in scheds:
            for flags in flags_list:
                p = W.Params(sched=sched, flags=flags)
                g.run(W.APP_BFS, p)
                got = g.read_results()
                helpers.check_bfs(got, V, s, d, 0, levels)
                assert parents is None or np.array_equal(got, parents), "parents differ between schedules"
                parents = got
                g.run(W.APP_CC, p)
                assert np.array_equal(g.read_results().view(np.float64), labels)
                g.run(W.APP_SSSP, p)
                assert np.array_equal(g.read_results(), dist)
                gf.run(W.APP_SSSP, p)
                got = gf.read_results()
                assert fdist is None or np.array_equal(got, fdist), "FP64 distances differ between schedules"
                fdist = got


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 127, 128, 129, 255, 257, 1023, 5000])
def test_out_lists_of_the_loop(engine_lib, n):
    """out-lists around what a warp takes at once (32 vertices, 128 out-edges), the
    whole traversal in one launch, iteration by iteration and host-driven"""
    W = engine_lib
    V, s, d, w = fan_in_out(n, n)
    check_traversals(W, V, s, d, w, (W.SCHED_PLAIN, W.SCHED_DENSE, W.SCHED_WEDGE, W.SCHED_FILTERED),
                     (0, W.FLAG_GRAPH, W.FLAG_TIMING))


@pytest.mark.parametrize("edges", [(1 << 20) - 513, 1 << 20, (1 << 20) + 1, (1 << 20) + 700])
def test_largest_whole_traversal(engine_lib, edges):
    """graphs around the size up to which a traversal is one launch; past it the dense
    iterations take their own launches"""
    W = engine_lib
    rng = np.random.default_rng(edges)
    V = 70_001
    # a short-diameter core and a long tail of vertices, so that every strategy runs
    core = rng.integers(0, 4000, (2, edges - 20_000))
    tail = np.arange(4000, 24_000)
    s = np.concatenate([core[0], np.where(tail % 50 == 0, tail % 4000, tail - 1)])
    d = np.concatenate([core[1], tail])
    order = np.lexsort((s, d))
    s, d = s[order].astype(np.uint32), d[order].astype(np.uint32)
    w = rng.integers(0, 256, len(s)).astype(np.uint64)
    check_traversals(W, V, s, d, w, (W.SCHED_PLAIN, W.SCHED_FILTERED), (0, W.FLAG_GRAPH, W.FLAG_TIMING))


@pytest.mark.parametrize("weights", ["bytes", "zeros", "words", "beyond32", "f64"])
def test_near_vertices_first(engine_lib, weights):
    """long SSSPs with many changed vertices, where far ones wait: the distances are
    those of all-dense pulls, whatever interrupts the loop (schedules, one
    iteration at a time), with zero weights, wide ones and 32-bit overflow"""
    W = engine_lib
    side, rng = 700, np.random.default_rng(5)
    v = np.arange(side * side).reshape(side, side)
    s = np.concatenate([v[:, :-1].ravel(), v[:, 1:].ravel(), v[:-1].ravel(), v[1:].ravel(), rng.integers(0, side * side, 9000)])
    d = np.concatenate([v[:, 1:].ravel(), v[:, :-1].ravel(), v[1:].ravel(), v[:-1].ravel(), rng.integers(0, side * side, 9000)])
    order = np.lexsort((s, d))
    s, d = s[order].astype(np.uint32), d[order].astype(np.uint32)
    n = len(s)
    kind = W.WEIGHTS_U64
    if weights == "f64":
        w, kind = rng.random(n).view(np.uint64), W.WEIGHTS_F64
    else:
        w = {"bytes": rng.integers(1, 256, n), "zeros": rng.integers(0, 2, n) * rng.integers(1, 256, n),
             "words": rng.integers(0, 100_000, n), "beyond32": rng.integers(0, 1 << 31, n)}[weights].astype(np.uint64)
    with W.Graph.from_edges(side * side, s, d, w, kind) as g:
        g.run(W.APP_SSSP, W.Params(sched=W.SCHED_DENSE))
        expect = g.read_results().copy()
        for sched in (W.SCHED_PLAIN, W.SCHED_WEDGE):
            for flags in (0, W.FLAG_GRAPH, W.FLAG_TIMING):
                st = g.run(W.APP_SSSP, W.Params(sched=sched, flags=flags))
                assert st["iterations"] > 32
                assert np.array_equal(g.read_results(), expect), (sched, flags)


def plain_pagerank(V, src, dst, iterations, damping):
    outdeg = np.bincount(src, minlength=V).astype(np.float64)
    outdeg[outdeg == 0] = V
    outdeg = outdeg.astype(np.longdouble)
    rank = (np.longdouble(1.0) / V) / outdeg
    for _ in range(iterations):
        acc = np.zeros(V, np.longdouble)  # a plain double sum of a hub's in-edges is off by more than the engine's
        np.add.at(acc, dst, rank[src])
        rank = ((acc + (1.0 - acc.sum()) / V) * damping + (1.0 - damping) / V) / outdeg
    return rank.astype(np.float64)


@pytest.mark.parametrize("iterations", [1, 2, 5])
@pytest.mark.parametrize("degrees", ["one", "tile", "hub", "mixed"])
def test_pagerank_in_one_launch(engine_lib, iterations, degrees):
    """in-degrees around the tiles (256 and 512 in-edges): a tile of 256 or more
    destinations, destinations that end with a tile, that span two, nine and more;
    vertices without in-edges, without out-edges and without both; odd and even
    iteration counts (double-buffered ranks), and the phases after a run"""
    W = engine_lib
    rng = np.random.default_rng(iterations)
    ind = {"one": np.ones(1500, np.int64), "tile": np.array([256, 512, 255, 1, 257, 511, 513, 256, 3, 253]),
           "hub": np.array([5, 700, 4607, 4608, 20_000, 1, 2560]), "mixed": rng.integers(0, 60, 900)}[degrees]
    V = len(ind) + 700
    d = np.repeat(np.arange(len(ind)), ind)
    s = rng.integers(len(ind) // 2, V - 50, len(d))
    order = np.lexsort((s, d))
    s, d = s[order].astype(np.uint32), d[order].astype(np.uint32)
    expect = plain_pagerank(V, s.astype(np.int64), d.astype(np.int64), iterations, 0.85)
    with W.Graph.from_edges(V, s, d) as g:
        for prec, tol in ((W.PREC_FP64, 1e-13), (W.PREC_FP32C, 1e-6)):
            for flags in (0, W.FLAG_GRAPH, W.FLAG_TIMING):
                p = W.Params(num_iterations=iterations, damping=0.85, precision=prec, flags=flags)
                st = g.run(W.APP_PR, p)
                got = g.read_results().view(np.float64).copy()
                assert np.abs(got - expect).sum() <= tol * np.abs(expect).sum()
                assert abs(st["pr_sum"] - 1.0) < 1e-6 and st["iterations"] == iterations
            # one more iteration by phases from the FP64 run's ranks
        g.run(W.APP_PR, W.Params(num_iterations=iterations, damping=0.85))
        p = W.Params(damping=0.85)
        g.run_phase(W.APP_PR, W.PHASE_PULL_DENSE, p)
        g.run_phase(W.APP_PR, W.PHASE_VERTEX_PR, p)
        more = plain_pagerank(V, s.astype(np.int64), d.astype(np.int64), iterations + 1, 0.85)
        assert np.abs(g.read_results().view(np.float64) - more).sum() <= 1e-13 * np.abs(more).sum()


@pytest.mark.parametrize("n", [1, 4, 5, 31, 33, 64, 65, 127, 128, 129, 513, 577, 9001])
@pytest.mark.parametrize("weights", ["bytes", "words", "f64"])
def test_batched_pulls(engine_lib, n, weights):
    """out- and in-lists around the batched kernel's sizes (lists of 128 out-edges
    and pieces of the longer ones, chunks of 4 listed vertices, groups of 32
    destinations of up to 64 in-edges, pieces of 512), all pulls sparse, all dense and mixed"""
    W = engine_lib
    V, s, d, w = fans(n, "random", n)
    kind = W.WEIGHTS_U64
    if weights == "words":
        w = w * np.uint64(1 << 20)
    elif weights == "f64":
        w, kind = (w.astype(np.float64) / 8.0).view(np.uint64), W.WEIGHTS_F64
    with W.Graph.from_edges(V, s, d, w, kind) as g:
        queries = [(0, app, root) for app in (W.APP_SSSP, W.APP_BFS) for root in (0, 1, n, V - 1)]
        expect = []
        for _, app, root in queries:
            g.run(app, W.Params(root=root, sched=W.SCHED_DENSE))
            expect.append(g.read_results().copy())
        if weights == "bytes":
            assert np.array_equal(expect[0], bellman_ford(V, s.astype(np.int64), d.astype(np.int64), w, 0))
        with W.Batch([g], queries) as b:
            for threshold_pct in (1, 20, 100):
                b.run(W.BatchTuning(threshold_pct=threshold_pct))
                for i, (_, app, root) in enumerate(queries):
                    got = b.read_result(i)
                    if app == W.APP_SSSP:
                        assert np.array_equal(got, expect[i]), (threshold_pct, root)
                    else:  # the targets' parents may be any middle vertex that was reached
                        none = np.uint64(0xFFFFFFFFFFFFFFFF)
                        assert np.array_equal(got == none, expect[i] == none)
                        assert np.array_equal(got[:n + 1], expect[i][:n + 1])
                        tail = got[n + 1:][got[n + 1:] != none].astype(np.int64)
                        assert np.all((tail == root) | ((tail >= 1) & (tail <= n)))


@pytest.mark.parametrize("late", [0, 1, 2, 15, 40])
@pytest.mark.parametrize("n", [1, 31, 33, 64, 300])
def test_first_sources(engine_lib, monkeypatch, n, late):
    """dense pulls that probe n destinations, each settled by its first source or by
    the one after `late` others (within the probe window and past it), where the
    launches run apart from the loop of small graphs"""
    W = engine_lib
    monkeypatch.setenv("WEDGE_CSRI_CHUNKS", "1")
    # 0 -> 1 -> n destinations; `late` vertices that nothing reaches, of more out-edges, point at all of them too
    V = 2 + n + late + 70
    dests, others, extra = np.arange(2, 2 + n), np.arange(2 + n, 2 + n + late), np.arange(2 + n + late, V)
    s = np.concatenate([[0], np.full(n, 1), np.repeat(others, n + 70)])
    d = np.concatenate([[1], dests, np.tile(np.concatenate([dests, extra]), late)])
    order = np.lexsort((s, d))
    s, d = s[order].astype(np.uint32), d[order].astype(np.uint32)
    none = np.uint64(0xFFFFFFFFFFFFFFFF)
    parents = np.full(V, none)
    parents[1], parents[dests] = 0, 1  # the root itself reads as without a parent
    for flags in (0, W.FLAG_GRAPH):
        with W.Graph.from_edges(V, s, d) as g:
            g.run(W.APP_BFS, W.Params(root=0, sched=W.SCHED_DENSE, flags=flags))
            assert np.array_equal(g.read_results(), parents)
            g.run(W.APP_CC, W.Params(sched=W.SCHED_DENSE, flags=flags))
            assert np.array_equal(g.read_results().view(np.float64), least_labels(V, s, d))
        both = np.lexsort((np.concatenate([s, d]), np.concatenate([d, s])))
        s2, d2 = np.concatenate([s, d])[both], np.concatenate([d, s])[both]
        with W.Graph.from_edges(V, s2, d2) as g:
            g.run(W.APP_CC, W.Params(sched=W.SCHED_DENSE, flags=flags))
            assert np.array_equal(g.read_results().view(np.float64), least_labels(V, s2, d2))


@pytest.mark.parametrize("limit", [None, 300])
@pytest.mark.parametrize("weights", ["bytes", "zeros", "equal", "steep"])
def test_bounded_weight_ordered_pulls(engine_lib, weights, limit):
    """several dense pulls in a row with a bound from the vertices the last one
    changed, Wedge iterations run as such pulls, and short tails after them, on a
    graph too large for the loop of small ones; a chain keeps a few vertices
    changing, and some sums pass a 32-bit limit"""
    W = engine_lib
    rng = np.random.default_rng(len(weights))
    V, n = 60_001, 1_250_000
    s = np.minimum((V * rng.random(n) ** 3).astype(np.int64), V - 2)
    d = np.minimum((V * rng.random(n) ** 2).astype(np.int64), V - 2)
    chain = rng.permutation(V - 1)[:300]
    s, d = np.concatenate([s, chain[:-1]]), np.concatenate([d, chain[1:]])
    w = {"bytes": rng.integers(0, 256, len(s)), "zeros": rng.integers(0, 256, len(s)) * (rng.random(len(s)) < 0.3),
         "equal": np.full(len(s), 7), "steep": np.minimum(255, s % 256 + 1)}[weights].astype(np.int64)
    w[-299:] = 1
    order = np.lexsort((s, d))
    s, d, w = s[order].astype(np.uint32), d[order].astype(np.uint32), w[order].astype(np.uint64)
    root = int(s[0])
    expect = bellman_ford(V, s, d, w, root)
    with W.Graph.from_edges(V, s, d, w) as g:
        g.set_knob("sssp_narrow", limit)
        for sched in (W.SCHED_PLAIN, W.SCHED_DENSE, W.SCHED_FILTERED, W.SCHED_WEDGE):
            for flags in (0, W.FLAG_GRAPH, W.FLAG_TIMING):
                for threshold_pct in (1, 20, 100):
                    g.run(W.APP_SSSP, W.Params(root=root, sched=sched, flags=flags, threshold_pct=threshold_pct))
                    assert np.array_equal(g.read_results(), expect), (sched, flags, threshold_pct)


@pytest.mark.parametrize("n", [100_000, 300_001])
def test_heavy_wedge_iterations(engine_lib, n):
    """BFS and CC with a frontier of many vertices of one out-edge each, below the
    dense threshold: too few and enough of them to run as a dense pull"""
    W = engine_lib
    rng = np.random.default_rng(n)
    middle, target = np.arange(1, n + 1), np.arange(n + 1, 2 * n + 1)
    V = 2 * n + 1001
    # 0 -> n vertices -> one more each, and edges among 1000 others that count towards the threshold
    s = np.concatenate([np.zeros(n, np.int64), middle, 2 * n + 1 + rng.integers(0, 1000, 3_000_000)])
    d = np.concatenate([middle, rng.permutation(target), 2 * n + 1 + rng.integers(0, 1000, 3_000_000)])
    order = np.lexsort((s, d))
    s, d = s[order], d[order]
    parents = np.full(V, np.uint64(0xFFFFFFFFFFFFFFFF))
    reached = (d <= 2 * n)
    parents[d[reached]] = s[reached]
    labels = least_labels(V, s, d)
    with W.Graph.from_edges(V, s.astype(np.uint32), d.astype(np.uint32)) as g:
        for sched in (W.SCHED_PLAIN, W.SCHED_WEDGE, W.SCHED_DENSE):
            for flags in (0, W.FLAG_GRAPH, W.FLAG_TIMING):
                st = g.run(W.APP_BFS, W.Params(root=0, sched=sched, flags=flags))
                assert st["iterations"] == 2  # the targets have no out-edges
                assert np.array_equal(g.read_results(), parents), (sched, flags)
                g.run(W.APP_CC, W.Params(sched=sched, flags=flags))
                assert np.array_equal(g.read_results().view(np.float64), labels), (sched, flags)


def sorted_again_and_again(filler, seed):
    """An SSSP whose far vertices become near and far again under a bound that falls: a
    path from 0 with fans of out-edges on it.  D (past the first 16 iterations) sets
    the first bound and leaves A, behind a long edge, beyond it; A is released and
    lowers the targets T, which have no out-edges, past the second bound; B lowers
    them below it; R ends the sorting with its fewer out-edges; C lowers T past the
    third bound, which is the least.  Returns the edges and the vertices of T."""
    T, path = 70_000, 40
    a, v0 = path + 1, path + 2  # vertices 0..path, A, then T and others that only receive
    junk = v0 + T
    V = junk + 40
    fan = {14: (20_000, 1), 15: (66_000, 1), 22: (20_000, 1)}  # path vertex -> out-edges to the others, weight
    parts = [(np.arange(path), np.arange(1, path + 1), np.ones(path, np.int64))]
    for p, (n, w) in fan.items():
        parts.append((np.full(n, p), junk + np.arange(n) % 40, np.full(n, w)))
    parts.append(([15], [a], [10_000_000]))
    for p, w in ((a, 4_000_000), (20, 5_000_000), (23, 4_000_000)):
        parts.append((np.full(T, p), v0 + np.arange(T), np.full(T, w)))
    rng = np.random.default_rng(seed)
    parts.append((junk + rng.integers(0, 20, filler), junk + 20 + rng.integers(0, 20, filler), rng.integers(0, 2, filler)))
    s, d, w = (np.concatenate([p[i] for p in parts]).astype(np.int64) for i in range(3))
    order = np.lexsort((s, d))
    return V, s[order], d[order], w[order], np.arange(v0, v0 + T)


def real_distances(V, src, dst, w, root):
    """least path sums in doubles, in the order of the path; inf = unreached"""
    dist = np.full(V, np.inf)
    dist[root] = 0.0
    while True:
        new = dist.copy()
        np.minimum.at(new, dst, dist[src] + w)
        if np.array_equal(new, dist):
            return dist
        dist = new


@pytest.mark.parametrize("places", [None, 1, 64, 70_000])
@pytest.mark.parametrize("filler", [100_000, 1_200_000])
@pytest.mark.parametrize("weights", ["words", "f64"])
def test_far_list_holds_a_vertex_once(engine_lib, monkeypatch, weights, filler, places):
    """vertices that are sorted out again and again, also with a list that fills up,
    in one launch (100,000 more edges) and apart from the dense pulls"""
    W = engine_lib
    if places is not None:
        monkeypatch.setenv("WEDGE_FAR_LIST", str(places))
    V, s, d, w, _ = sorted_again_and_again(filler, 1)
    if weights == "f64":
        expect, words, kind = real_distances(V, s, d, w + 0.25, 0).view(np.uint64), (w + 0.25).view(np.uint64), W.WEIGHTS_F64
    else:
        expect, words, kind = bellman_ford(V, s, d, w, 0), w.astype(np.uint64), W.WEIGHTS_U64
    with W.Graph.from_edges(V, s.astype(np.uint32), d.astype(np.uint32), words, kind) as g:
        for sched in (W.SCHED_PLAIN, W.SCHED_WEDGE):
            for flags in (0, W.FLAG_GRAPH):
                g.run(W.APP_SSSP, W.Params(sched=sched, flags=flags))
                assert np.array_equal(g.read_results(), expect), (sched, flags)


@pytest.mark.parametrize("places", [None, 1, 1000])
def test_far_list_of_a_grid(engine_lib, monkeypatch, places):
    """the same on a grid with random pairs, against plain arithmetic"""
    W = engine_lib
    if places is not None:
        monkeypatch.setenv("WEDGE_FAR_LIST", str(places))
    side, rng = 700, np.random.default_rng(8)
    v = np.arange(side * side).reshape(side, side)
    s = np.concatenate([v[:, :-1].ravel(), v[:, 1:].ravel(), v[:-1].ravel(), v[1:].ravel(), rng.integers(0, side * side, 9000)])
    d = np.concatenate([v[:, 1:].ravel(), v[:, :-1].ravel(), v[1:].ravel(), v[:-1].ravel(), rng.integers(0, side * side, 9000)])
    order = np.lexsort((s, d))
    s, d, w = s[order], d[order], rng.integers(0, 100_000, len(s))
    expect = bellman_ford(side * side, s, d, w, 0)
    with W.Graph.from_edges(side * side, s.astype(np.uint32), d.astype(np.uint32), w.astype(np.uint64)) as g:
        for flags in (0, W.FLAG_GRAPH):
            g.run(W.APP_SSSP, W.Params(flags=flags))
            assert np.array_equal(g.read_results(), expect), flags


def rounds_of_all_changed(V, src, dst, w, root):
    """distances, and the iterations in which every vertex changed by the last one relaxes its out-edges"""
    dist = np.full(V, 1 << 62, np.int64)
    dist[root] = 0
    n = 0
    while True:
        new = dist.copy()
        reached = dist[src] < 1 << 62
        np.minimum.at(new, dst[reached], dist[src[reached]] + w[reached])
        if np.array_equal(new, dist):
            return np.where(dist >= 1 << 62, np.uint64(0xFFFFFFFFFFFFFFFF), dist.astype(np.uint64)), n
        dist, n = new, n + 1


@pytest.mark.parametrize("graph", ["grid", "steps"])
def test_iteration_caps_of_long_sssp(engine_lib, graph):
    """a cap that suffices when every changed vertex is visited at once suffices, and
    one that does not is kept to; no cap is |V| + 1, which always suffices: "steps" is
    a path whose shortcuts change nearly all vertices in nearly |V| iterations"""
    W = engine_lib
    rng = np.random.default_rng(3)
    if graph == "grid":
        side = 700
        V = side * side
        v = np.arange(V).reshape(side, side)
        s = np.concatenate([v[:, :-1].ravel(), v[:, 1:].ravel(), v[:-1].ravel(), v[1:].ravel(), rng.integers(0, V, 9000)])
        d = np.concatenate([v[:, 1:].ravel(), v[:, :-1].ravel(), v[1:].ravel(), v[:-1].ravel(), rng.integers(0, V, 9000)])
        w = rng.integers(1, 100_000, len(s))
    else:
        V = 120
        i, j = np.triu_indices(V, 1)
        copies = 200  # 1.4 M edges, most of them parallel
        s, d = np.repeat(i, copies), np.repeat(j, copies)
        w = np.repeat(np.where(j == i + 1, 1, 300 * (j - i)), copies)
    order = np.lexsort((s, d))
    s, d, w = s[order], d[order], w[order].astype(np.int64)
    expect, rounds = rounds_of_all_changed(V, s, d, w, 0)
    with W.Graph.from_edges(V, s.astype(np.uint32), d.astype(np.uint32), w.astype(np.uint64)) as g:
        for sched in (W.SCHED_PLAIN, W.SCHED_WEDGE):
            for flags in (0, W.FLAG_GRAPH):
                for cap in (0, rounds + 1):
                    st = g.run(W.APP_SSSP, W.Params(sched=sched, flags=flags, max_iterations=cap))
                    assert cap == 0 or st["iterations"] <= cap
                    assert np.array_equal(g.read_results(), expect), (sched, flags, cap)
                st = g.run(W.APP_SSSP, W.Params(sched=sched, flags=flags, max_iterations=30), allow_not_converged=True)
                assert st["iterations"] == 30, (sched, flags)


@pytest.mark.parametrize("weights", ["none", "bytes", "f64"])
def test_loads_with_little_memory(engine_lib, weights):
    """a load takes the optional copies of the in-edges and the out-edges' arrays only
    where they fit: it succeeds from what the sort of the in-edges needs (the edges
    and their sort keys, twice, and the vertices' arrays), and says so below it"""
    import torch

    W = engine_lib
    rng = np.random.default_rng(1)
    V, n = 1 << 20, (1 << 23) - 5000
    s = np.minimum((V * rng.random(n) ** 2).astype(np.int64), V - 1)
    d = np.sort(np.minimum((V * rng.random(n) ** 3).astype(np.int64), V - 1))
    s[:2], d[:2] = (0, 1), (0, 0)
    s, d = s.astype(np.uint32), d.astype(np.uint32)
    args, app, per_edge = (), W.APP_BFS, 24
    if weights == "bytes":
        args, app, per_edge = (rng.integers(0, 256, n).astype(np.uint64),), W.APP_SSSP, 40
    elif weights == "f64":
        args, app, per_edge = (rng.random(n).view(np.uint64), W.WEIGHTS_F64), W.APP_SSSP, 40
    root = int(s[n // 2])
    need = per_edge * n + 64 * V + (48 << 20)
    expect = None
    outcomes = []
    for room in (need + (1 << 30), need + (96 << 20), need + (48 << 20), need, need // 2, need // 8):
        torch.cuda.empty_cache()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        held = torch.empty(free - room, dtype=torch.uint8, device="cuda")
        try:
            g = W.Graph.from_edges(V, s, d, *args)
        except W.WedgeError as e:
            outcomes.append((room, e.status))
            g = None
        del held
        torch.cuda.empty_cache()
        if g is not None:
            with g:
                g.run(app, W.Params(root=root))
                got = g.read_results()
                outcomes.append((room, 0))
            if expect is None:
                expect = got
            if app == W.APP_BFS:  # parents may be others: the same vertices are reached
                got, expect = got == np.uint64(0xFFFFFFFFFFFFFFFF), expect == np.uint64(0xFFFFFFFFFFFFFFFF) \
                    if expect.dtype == np.uint64 else expect
            assert np.array_equal(got, expect), room
    assert [rc for room, rc in outcomes if room >= need] == [0] * 4, outcomes
    assert outcomes[-1][1] == W.engine.ERR_OOM, outcomes
    with W.Graph.from_edges(V, s, d, *args) as g:  # nothing of the failed loads is left
        g.run(app, W.Params(root=root))


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("n", [900, 40_000])
def test_asked_strategies_of_small_graphs(engine_lib, n, symmetric):
    """a strategy that a caller asks for is the one that runs, on a graph of any size
    (dense pulls are launches of their own, Wedge iterations share one), and the
    results are the plain rule's"""
    W = engine_lib
    rng = np.random.default_rng(n)
    V = n // 2
    s, d = rng.integers(0, V, n), (V * rng.random(n) ** 2).astype(np.int64)
    if symmetric:
        s, d = np.concatenate([s, d]), np.concatenate([d, s])
    order = np.lexsort((s, d))
    s, d = s[order].astype(np.uint32), d[order].astype(np.uint32)
    w = rng.integers(0, 256, len(s)).astype(np.uint64)
    check_traversals(W, V, s, d, w, (W.SCHED_PLAIN, W.SCHED_DENSE, W.SCHED_WEDGE, W.SCHED_FILTERED), (0, W.FLAG_GRAPH))
    with W.Graph.from_edges(V, s, d, w) as g:
        for app in (W.APP_BFS, W.APP_CC, W.APP_SSSP):
            launches = {}
            for sched in (W.SCHED_PLAIN, W.SCHED_DENSE, W.SCHED_FILTERED):
                st = g.run(app, W.Params(sched=sched, flags=W.FLAG_GRAPH))
                launches[sched] = st["kernel_launches"]
            # preparation (2), the loop, CC's labels (2); else a dense iteration's pulls and decision as well
            assert launches[W.SCHED_PLAIN] <= 5 < min(launches[W.SCHED_DENSE], launches[W.SCHED_FILTERED]), launches


@pytest.mark.parametrize("n", [100_000, 300_001])
def test_log_says_which_pulls_ran(engine_lib, n):
    """the iterations' log of timed, captured and host-driven runs: a frontier too large
    for its out-edges one by one is a dense pull in all of them, and reads as one"""
    W = engine_lib
    rng = np.random.default_rng(n)
    V = 2 * n + 1001
    s = np.concatenate([np.zeros(n, np.int64), np.arange(1, n + 1), 2 * n + 1 + rng.integers(0, 1000, 3_000_000)])
    d = np.concatenate([np.arange(1, n + 1), n + 1 + rng.permutation(n), 2 * n + 1 + rng.integers(0, 1000, 3_000_000)])
    order = np.lexsort((s, d))
    with W.Graph.from_edges(V, s[order].astype(np.uint32), d[order].astype(np.uint32)) as g:
        logs = []
        for flags in (0, W.FLAG_GRAPH, W.FLAG_TIMING):
            st = g.run(W.APP_BFS, W.Params(root=0, flags=flags))
            log = g.iteration_log()
            assert [r["mode"] for r in log] == [W.MODE_WEDGE, W.MODE_DENSE if n > 200_000 else W.MODE_WEDGE]
            assert st["wedge_iterations"] == sum(r["used_wedge"] for r in log) == sum(r["mode"] == W.MODE_WEDGE for r in log)
            logs.append([(r["mode"], r["active_edges"], r["changed_mass"], r["vertices_activated"]) for r in log])
            if flags == W.FLAG_TIMING:
                assert all(r["pull_ms"] > 0.0 for r in log)
        assert logs[0] == logs[1] == logs[2]


@pytest.mark.parametrize("graph", ["grid", "rmat18", "rmat12"])
def test_timed_runs_are_the_plain_runs(engine_lib, graph):
    """a run with per-iteration times takes the kernels that a run without takes: far
    vertices wait in it, PageRank is one launch, and the times add up to the run's"""
    W = engine_lib
    make = {"grid": lambda wk: W.Graph.grid(1500, 0.01, 5, wk), "rmat18": lambda wk: W.Graph.rmat(18, 16, 5, weight_kind=wk),
            "rmat12": lambda wk: W.Graph.rmat(12, 16, 5, weight_kind=wk)}[graph]
    with make(W.WEIGHTS_U64) as g:
        for app in (W.APP_SSSP, W.APP_BFS, W.APP_CC):
            plain = g.run(app, W.Params(flags=W.FLAG_GRAPH))
            expect = g.read_results().copy()
            for _ in range(2):
                st = g.run(app, W.Params(flags=W.FLAG_TIMING))
            assert app == W.APP_BFS or np.array_equal(g.read_results(), expect)
            log = g.iteration_log()
            assert st["edges_scanned"] <= 1.5 * plain["edges_scanned"] and plain["edges_scanned"] <= 1.5 * st["edges_scanned"]
            assert len(log) == st["iterations"] and all(r["pull_ms"] >= 0.0 and r["wedge_ms"] >= 0.0 for r in log)
            total = st["pull_ms_dense"] + st["pull_ms_wedge"] + st["wedge_ms"]
            assert abs(sum(r["pull_ms"] + r["wedge_ms"] for r in log) - total) < 1e-3 * total
            assert total < st["running_ms"]
            if plain["running_ms"] > 1.0:  # the launches around the iterations are little beside them
                assert total > 0.6 * plain["running_ms"], (total, plain["running_ms"])
        for prec in (W.PREC_FP64, W.PREC_FP32C):
            p = dict(num_iterations=7, damping=0.85, precision=prec)
            plain = g.run(W.APP_PR, W.Params(**p))
            expect = g.read_results().copy()
            st = g.run(W.APP_PR, W.Params(flags=W.FLAG_TIMING, **p))
            assert np.array_equal(g.read_results(), expect)
            assert st["pull_launches"] == plain["pull_launches"] == 1 and st["kernel_launches"] == 1
            log = g.iteration_log()
            assert len(log) == 7 and all(r["pull_ms"] > 0.0 for r in log)
            assert 0.0 < sum(r["pull_ms"] for r in log) + st["vertex_ms"] < st["running_ms"]


def test_captured_loops_without_cooperative_launches(engine_lib, monkeypatch):
    """under MPS a captured loop's iterations are separate launches: the results are the
    host-driven loop's, and so are those of small graphs, which are no captured loop"""
    W = engine_lib
    monkeypatch.setenv("WEDGE_MPS", "1")
    rng = np.random.default_rng(12)
    for n in (60_000, 1_200_000):
        V = n // 8
        s, d = (V * rng.random(n) ** 2).astype(np.int64), (V * rng.random(n) ** 2).astype(np.int64)
        s, d = np.concatenate([s, np.arange(200)]), np.concatenate([d, np.arange(1, 201)])
        order = np.lexsort((s, d))
        w = rng.integers(0, 256, len(s)).astype(np.uint64)
        check_traversals(W, V, s[order].astype(np.uint32), d[order].astype(np.uint32), w,
                         (W.SCHED_PLAIN, W.SCHED_WEDGE, W.SCHED_FILTERED), (0, W.FLAG_GRAPH, W.FLAG_TIMING))


@pytest.mark.parametrize("iterations", [1, 2, 7])
def test_vertex_phase_after_a_pagerank(engine_lib, iterations):
    """the vertex phase alone after a run works on the run's last sums: the same ranks
    with the same damping, that iteration's with another"""
    W = engine_lib
    rng = np.random.default_rng(iterations)
    V, n = 3000, 40_000
    s, d = (V * rng.random(n) ** 3).astype(np.int64), np.sort((V * rng.random(n) ** 2).astype(np.int64))
    s[-1], s, d = V - 5, s.astype(np.uint32), d.astype(np.uint32)
    outdeg = np.bincount(s, minlength=V).astype(np.float64)
    outdeg[outdeg == 0] = V
    before = plain_pagerank(V, s.astype(np.int64), d.astype(np.int64), iterations - 1, 0.85)
    acc = np.zeros(V, np.longdouble)
    np.add.at(acc, d, before.astype(np.longdouble)[s])
    with W.Graph.from_edges(V, s, d) as g:
        g.run(W.APP_PR, W.Params(num_iterations=iterations, damping=0.85))
        ran = g.read_results().view(np.float64).copy()
        for damping in (0.85, 0.6, 0.85):
            g.run_phase(W.APP_PR, W.PHASE_VERTEX_PR, W.Params(damping=damping))
            got = g.read_results().view(np.float64)
            expect = (((acc + (1.0 - acc.sum()) / V) * damping + (1.0 - damping) / V) / outdeg).astype(np.float64)
            assert np.abs(got - expect).sum() <= 1e-13 * np.abs(expect).sum(), damping
        assert np.abs(got - ran).sum() <= 1e-13 * np.abs(ran).sum()


def test_timed_runs_past_the_log(engine_lib):
    """more iterations than the log keeps: the kept ones have their own times, the
    others' are in the totals"""
    W = engine_lib
    V = 6001
    s, d = np.arange(V - 1, dtype=np.uint32), np.arange(1, V, dtype=np.uint32)
    with W.Graph.from_edges(V, s, d) as g:
        for app, p in ((W.APP_BFS, {}), (W.APP_PR, dict(num_iterations=6000))):
            for _ in range(2):
                st = g.run(app, W.Params(flags=W.FLAG_TIMING, **p))
            times = np.array([r["pull_ms"] for r in g.iteration_log()])
            total = st["pull_ms_dense"] + st["pull_ms_wedge"] + st["vertex_ms"]
            assert st["iterations"] == 6000 and len(times) == 4096
            assert times.min() > 0.0 and times[0] < 50 * np.median(times)
            assert 0.8 * st["running_ms"] < total <= st["running_ms"] and total > 1.3 * times.sum()
