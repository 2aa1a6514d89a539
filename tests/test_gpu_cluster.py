"""The cluster frontier loops: pieces of long lists, queues that spill, small and large exits."""
import numpy as np
import pytest

import cggraph_b200 as cg
from oracle import oracle as O

BFS, SSSP = int(cg.Algorithm_type.BFS), int(cg.Algorithm_type.SSSP)


def csr(V, src, dst, seed, wmax):
    key = np.unique(src.astype(np.int64) * V + dst)
    src, dst = key // V, (key % V).astype(np.uint32)
    off = np.zeros(V + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(src, minlength=V))
    w = np.random.default_rng(seed).integers(1, wmax + 1, dst.size).astype(np.uint32)
    return off, dst, w


def star(leaves, degree):
    """Vertex 0 to every leaf, each leaf to `degree` others: the second frontier has leaves * ceil(degree / 8) pieces."""
    V = leaves + 1
    i = np.repeat(np.arange(1, V), degree)
    j = (i * 7 + 13 * np.tile(np.arange(degree), leaves)) % V
    return V, np.concatenate([np.zeros(leaves, np.int64), i]), np.concatenate([np.arange(1, V), j])


def ladder(degrees):
    """A chain whose i-th vertex also points at degrees[i] leaves: lists around the piece size, thin frontiers."""
    n = len(degrees)
    src, dst, nxt = [], [], n
    for i, d in enumerate(degrees):
        if i + 1 < n:
            src.append(i), dst.append(i + 1)
        src += [i] * d
        dst += range(nxt, nxt + d)
        nxt += d
    return nxt, np.array(src), np.array(dst)


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [
    lambda: star(100_000, 9),     # the queues spill
    lambda: star(65_000, 8),      # one piece a leaf, a queue nearly full
    lambda: star(160_000, 2),     # more far vertices than the cluster splits
    lambda: star(3, 2),
    lambda: ladder([0, 1, 6, 7, 8, 9, 14, 15, 16, 17, 30, 31, 32, 33, 255, 256, 257, 5000] * 3),
])
@pytest.mark.parametrize("wmax,delta", [(1, 0), (1000, 0), (1000, 50)])
def test_cluster_loops(graph, wmax, delta):
    V, src, dst = graph()
    keep = src != dst
    off, dst, w = csr(V, src[keep], dst[keep], 5, wmax)
    # the tail without out-edges is left out of the frontiers
    nz = int(np.nonzero(np.diff(off.astype(np.int64)))[0].max()) + 1
    with cg.Graph.from_csr(off, dst, w, noZeroOutDegreeNum=nz) as g:
        np.testing.assert_array_equal(g.run(BFS, 0)[0], O.bfs(off, dst, 0))
        opts = cg.make_options(sssp_delta=delta)
        np.testing.assert_array_equal(g.run(SSSP, 0, opts)[0], O.sssp(off, dst, w, 0))
        # again after the other algorithm used the shared scratch, from a vertex inside
        np.testing.assert_array_equal(g.run(BFS, 1)[0], O.bfs(off, dst, 1))
        np.testing.assert_array_equal(g.run(SSSP, 1, opts)[0], O.sssp(off, dst, w, 1))
    with cg.Graph.from_csr(off, dst) as g:  # unit weights
        np.testing.assert_array_equal(g.run(SSSP, 0)[0], O.bfs(off, dst, 0))


@pytest.mark.gpu
def test_wait_for_counts_ends():
    """A CTA that keeps its counts back ends the others' waits after their time limit, and the context stays usable."""
    import ctypes
    import time
    from cggraph_b200 import _lib as L
    f = L.lib().cgb_check_cluster_timeout
    f.argtypes = [ctypes.c_int, ctypes.c_uint32]
    f.restype = ctypes.c_int
    assert f(0, 0) == L.EINVAL and f(0, 1_000_001) == L.EINVAL
    assert f(0, 100) == L.ETIMEOUT
    t0 = time.monotonic()
    assert f(0, 200_000) == L.ETIMEOUT
    # the wait and, before the cluster leaves, once more as long
    assert 0.2 <= time.monotonic() - t0 < 5
    V, src, dst = ladder([3] * 40)
    off, dst, w = csr(V, src, dst, 5, 9)
    with cg.Graph.from_csr(off, dst, w) as g:
        np.testing.assert_array_equal(g.run(BFS, 0)[0], O.bfs(off, dst, 0))
        np.testing.assert_array_equal(g.run(SSSP, 0)[0], O.sssp(off, dst, w, 0))


def spill_twice(members, longs, long_deg):
    """A round that queues nearly every vertex again, more than the cluster's queues hold.  The root reaches `members`
    vertices with short lists at random distances and a hub at distance 1; a member's list names one vertex with a long
    list first (these fill the queues), then three members; the hub's list, expanded last, improves every member."""
    rng = np.random.default_rng(7)
    V = 1 + longs + members + 1
    first, hub = 1 + longs, V - 1
    m = np.arange(first, hub)
    a, b = np.repeat(m, 3), first + rng.integers(0, members, 3 * members)
    ls = np.repeat(np.arange(1, first), long_deg)
    ld = first + (np.arange(longs * long_deg) * 13) % members
    src = np.concatenate([np.zeros(members + 1, np.int64), m, a, ls, np.full(members, hub)])
    dst = np.concatenate([np.arange(first, V), 1 + np.arange(members) % longs, b, ld, m])
    return V, src[src != dst], dst[src != dst]


@pytest.mark.gpu
def test_spilled_vertex_leaves_once():
    """All vertices but two are in one round's next frontier, so a queue of V entries has no room for one of them twice."""
    V, src, dst = spill_twice(12_000, 4_096, 1_024)
    off, dd, _ = csr(V, src, dst, 5, 1)
    w = np.ones(dd.size, np.uint32)
    w[:off[1]] = np.random.default_rng(3).integers(1 << 16, 1 << 20, off[1])  # the root's edges,
    w[off[1] - 1] = 1                                                         # but for the hub's
    exp = O.sssp(off, dd, w, 0)
    with cg.Graph.from_csr(off, dd, w) as g:
        for _ in range(5):
            np.testing.assert_array_equal(g.run(SSSP, 0, cg.make_options(sssp_delta=1 << 30))[0], exp)


@pytest.mark.gpu
def test_spilled_hub_is_the_longest_list():
    """A frontier whose longest list left for the global queue is kept from the grid loop, which takes lists below
    persist_deg: seven hubs found by one thread, six fill a CTA's queue and the seventh, the longest, spills."""
    hubs = [9_600] * 6 + [20_000]
    leaves, each = sum(hubs), 62
    first, V = 1 + len(hubs), 1 + len(hubs) + leaves
    leaf = np.arange(first, V)
    src = np.concatenate([np.zeros(len(hubs), np.int64), np.repeat(np.arange(1, first), hubs), np.repeat(leaf, each)])
    dst = np.concatenate([np.arange(1, first), leaf, first + (np.arange(leaves * each) * 17 + 5) % leaves])
    off, dd, _ = csr(V, src, dst, 1, 1)
    assert np.diff(off[1:first + 1].astype(np.int64)).tolist() == hubs
    # the hubs' lists stay far from the direction switch, so that the grid loop is in question
    assert 4 * 15 * leaves < dd.size
    exp, launches = O.bfs(off, dd, 0), {}
    with cg.Graph.from_csr(off, dd) as g:
        for deg in (8_000, 16_000, 65_536):
            g.set_tuning({"persist_deg": deg})
            np.testing.assert_array_equal(g.run(BFS, 0)[0], exp)
            launches[deg] = g.stats().launches
    assert launches[8_000] == launches[16_000] != launches[65_536]


@pytest.mark.gpu
@pytest.mark.parametrize("leaves,degree", [(200_000, 6), (300_000, 4)])
def test_root_beyond_the_cluster_pulls(leaves, degree):
    """A root with more than a fifteenth of the edges is pulled from, as the direction rule has it, though the cluster
    loop was asked first and its out-edges were not known then."""
    V, src, dst = star(leaves, degree)
    off, dd, _ = csr(V, src[src != dst], dst[src != dst], 5, 1)
    root_edges = int(off[1])
    assert dd.size > 1 << 20 and 15 * root_edges > dd.size  # not a whole run in the cluster; beyond the switch point
    exp, pulls = O.bfs(off, dd, 0), []
    with cg.Graph.from_csr(off, dd) as g:
        for tuning in ({}, {"cluster_enter": 0}):
            g.set_tuning(tuning)
            np.testing.assert_array_equal(g.run(BFS, 0)[0], exp)
            s = g.stats()
            pulls.append((s.pulls_bu, s.pushes_td))
    assert pulls[0] == pulls[1] and pulls[0][0] > 0


@pytest.mark.gpu
def test_learned_delta_sees_vertices_not_pieces():
    """At the first bucket boundary the network is told how many vertices have been expanded, in the cluster as by the
    host's rounds: nine here (the root and eight hubs), whose lists are 2001 pieces.  A hand-made network picks four
    times the width when they are more than a two-hundredth of the vertices."""
    import torch
    from cggraph_b200 import _lib as L, policy
    hubs, leaves, fill, each = 8, 2_000, 1 << 16, 1 << 10  # the filler brings the edges to where the network is asked
    first = 1 + hubs + hubs * leaves
    V = first + fill
    dev = dict(device="cuda", dtype=torch.int32)
    deg = torch.tensor([hubs] + [leaves] * hubs + [0] * (hubs * leaves) + [each] * fill, **dev)
    off = torch.zeros(V + 1, **dev)
    off[1:] = deg.cumsum(0)
    dst = torch.cat([torch.arange(1, first, **dev), (first + torch.arange(each, **dev)).repeat(fill)])
    w = torch.full_like(dst, 64)
    w[:hubs] = 1
    w[hubs:hubs + hubs * leaves] = 1000
    p = np.zeros(policy.NP, np.float32)
    w1, w2, w3 = 0, 24 * 64 + 64, 24 * 64 + 64 + 64 * 64 + 64
    p[w1 + 23 * 64] = 1000.0    # settled / V
    p[24 * 64] = -5.0
    p[w2] = 1.0
    p[w3 + policy.SSSP_DELTA[4]] = -1.0
    p[w3 + 64 * 14:] = 1.0
    exp = np.full(V, cg.VALUE_MAX, np.uint32)
    exp[0], exp[1:1 + hubs], exp[1 + hubs:first] = 0, 1, 1001
    deltas = []
    policy.load(p)
    try:
        with cg.Graph.from_csr(off, dst, w, vertexNum=V, edgeNum=dst.numel()) as g:
            for tuning in ({"cluster_enter": 0}, {"cluster_enter": 8192}):
                g.set_tuning(tuning)
                np.testing.assert_array_equal(g.run(SSSP, 0, cg.make_options(schedule=L.SCHED_LEARNED))[0], exp)
                deltas.append(g.stats().sssp_delta)
            g.run(SSSP, 0)
            deltas.append(g.stats().sssp_delta)
    finally:
        policy.load(None)
    assert deltas[0] == deltas[1] == deltas[2] < 1000


@pytest.mark.gpu
@pytest.mark.parametrize("weight,factor", [(None, 128), (1, 128), (7, 128), ("mixed", 64)])
def test_default_width_of_large_meshes(weight, factor):
    """Graphs of 2^19 vertices or more without hubs: narrower default buckets only where edge lengths differ."""
    rows, cols = 725, 724
    with cg.Graph.grid(rows, cols, seed=1, wmax=1) as g:
        off, dst, _ = g.download(False)
    w = None
    if weight == "mixed":
        w = np.random.default_rng(2).integers(1, 1001, dst.size).astype(np.uint32)
        w[0] += 1 if w.sum(dtype=np.uint64) % dst.size == 0 else 0
    elif weight:
        w = np.full(dst.size, weight, np.uint32)
    mean = 1.0 if w is None else w.sum(dtype=np.uint64) / dst.size
    root = rows * cols // 2
    with cg.Graph.from_csr(off, dst, w) as g:
        got, _ = g.run(SSSP, root)
        assert g.stats().sssp_delta == int(factor * mean / (dst.size / (rows * cols)))
    exp = O.bfs(off, dst, root) * (weight or 1) if weight != "mixed" else O.sssp(off, dst, w, root)
    np.testing.assert_array_equal(got, exp)


@pytest.mark.gpu
@pytest.mark.parametrize("V,edges,pulls", [
    (2048, (1 << 19), False),      # the largest graph that runs in the cluster from start to end
    (2048, (1 << 19) + 1, True),   # and the smallest that does not: dense, most of it is pulled
    (2048, 900_000, True),
    (1 << 18, (1 << 19) + 1, None),
])
def test_whole_runs_in_the_cluster(V, edges, pulls):
    rng = np.random.default_rng(V + edges)
    key = np.unique(np.concatenate([np.arange(V, dtype=np.int64) * V + (np.arange(V) + 1) % V,
                                    rng.integers(0, V, 2 * edges) * V + rng.integers(0, V, 2 * edges)]))
    key = key[key // V != key % V]
    key = np.sort(rng.permutation(key)[:edges])
    off, dd, w = csr(V, key // V, key % V, 3, 20)
    assert dd.size == edges
    roots = np.nonzero(np.diff(off.astype(np.int64)))[0][[0, 7, -1]]
    with cg.Graph.from_csr(off, dd, w) as g:
        for r in map(int, roots):
            np.testing.assert_array_equal(g.run(BFS, r)[0], O.bfs(off, dd, r))
            if pulls is not None:
                assert (g.stats().pulls_bu > 0) == pulls
            np.testing.assert_array_equal(g.run(SSSP, r)[0], O.sssp(off, dd, w, r))


@pytest.mark.gpu
@pytest.mark.parametrize("hub", [65_535, 65_536, 65_537, 150_000])
def test_list_as_long_as_a_queue(hub):
    """A hub with as many edges as a CTA's queue holds, and more, found from a leaf: the loop is asked once for a list
    that it cannot hold, in a graph small enough to run there from start to end."""
    V = hub + 1
    src = np.concatenate([np.zeros(hub, np.int64), np.arange(1, V)])
    dst = np.concatenate([np.arange(1, V), np.zeros(hub, np.int64)])
    off, dd, w = csr(V, src, dst, 4, 50)
    assert dd.size <= 1 << 19
    with cg.Graph.from_csr(off, dd, w) as g:
        for root in (5, 0):
            np.testing.assert_array_equal(g.run(BFS, root)[0], O.bfs(off, dd, root))
            np.testing.assert_array_equal(g.run(SSSP, root)[0], O.sssp(off, dd, w, root))
        g.run(BFS, 5)
        launches = g.stats().launches
        g.set_tuning({"cluster_enter": 0})
        g.run(BFS, 5)
        # the loop's launch stands for the root's level (three launches) and is not followed by another
        assert launches <= (g.stats().launches if hub > 1 << 16 else 2)
