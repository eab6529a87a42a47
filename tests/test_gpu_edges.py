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
