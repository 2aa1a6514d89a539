"""The push expansion's staged queues and chunk descriptors at their edges, and bottom-up levels beside them."""
import numpy as np
import pytest

import cggraph_b200 as cg
from oracle import oracle as O

BFS, SSSP = int(cg.Algorithm_type.BFS), int(cg.Algorithm_type.SSSP)


def fan(first, second, seed):
    """Vertex 0 to `first` vertices; the i-th of those to second[i % len(second)] vertices of a wide last layer."""
    rng = np.random.default_rng(seed)
    deg = np.array([second[i % len(second)] for i in range(first)])
    last = max(1000, int(deg.sum() // 3))
    V = 1 + first + last
    src = np.concatenate([np.zeros(first, np.int64), np.repeat(np.arange(1, first + 1), deg)])
    dst = np.concatenate([np.arange(1, first + 1), 1 + first + rng.integers(0, last, int(deg.sum()))])
    key = np.unique(src * V + dst)
    src, dst = key // V, (key % V).astype(np.uint32)
    off = np.zeros(V + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(src, minlength=V))
    return off, dst, rng.integers(1, 65, dst.size).astype(np.uint32)


@pytest.mark.gpu
@pytest.mark.parametrize("first,second", [
    (40_000, [1, 2, 31, 32, 33]),            # more than 32768 vertices: the binned tiers
    (1_200, [3000, 255, 256, 257, 511, 512, 513, 1025]),  # chunked lists, many finds a warp
    (37, [60_000, 1, 0, 31]),                # a few hubs
    (33_000, [0, 0, 0, 200]),
])
@pytest.mark.parametrize("tuning", [{"push_block": 128}, {"push_block": 256}, {"push_block": 512}])
def test_push_edges(first, second, tuning):
    off, dst, w = fan(first, second, first)
    exp_b, exp_s = O.bfs(off, dst, 0), O.sssp(off, dst, w, 0)
    with cg.Graph.from_csr(off, dst, w) as g:
        # the host loop's kernels only; pushed levels, then the direction rule, then pulled ones
        g.set_tuning({"persist_enter": 0, "cluster_enter": 0, **tuning})
        for o in (cg.make_options(schedule=2, variant=3), None, cg.make_options(schedule=2, variant=2)):
            np.testing.assert_array_equal(g.run(BFS, 0, o)[0], exp_b)
        for alpha in (0, 4, 1024):  # no dense rounds, the default, every round dense
            g.set_tuning({"sssp_dense_alpha": alpha, "persist_enter": 0, "cluster_enter": 0, **tuning})
            np.testing.assert_array_equal(g.run(SSSP, 0)[0], exp_s)
        s = g.stats()
        assert s.reached == np.count_nonzero(exp_s != cg.VALUE_MAX)
        assert s.traversed_edges == int(np.diff(off.astype(np.int64))[exp_s != cg.VALUE_MAX].sum())


@pytest.mark.gpu
@pytest.mark.parametrize("first,second", [
    (1, [40_000]),                          # fewer chunks than CTAs: each is cut over a CTA's warps
    (90, [255, 256, 257, 288, 289, 31, 32, 33]),
    (1_183, [33, 64, 100, 256]),            # about as many chunks as CTAs (8 a SM), one below, one above
    (1_184, [256]),
    (1_185, [257]),
])
@pytest.mark.parametrize("block", [128, 256, 512])
def test_few_chunks(first, second, block):
    off, dst, w = fan(first, second, first + len(second))
    exp_b, exp_s = O.bfs(off, dst, 0), O.sssp(off, dst, w, 0)
    with cg.Graph.from_csr(off, dst, w) as g:
        g.set_tuning({"persist_enter": 0, "cluster_enter": 0, "push_block": block})
        np.testing.assert_array_equal(g.run(BFS, 0, cg.make_options(schedule=2, variant=3))[0], exp_b)
        np.testing.assert_array_equal(g.run(SSSP, 0)[0], exp_s)
        np.testing.assert_array_equal(g.run_batch(BFS, [0, 1])[0][0], exp_b)


@pytest.mark.gpu
@pytest.mark.parametrize("block", [128, 256, 512])
def test_binned_tiers(block):
    """A frontier above 2^19 vertices keeps the degree tiers: lists of up to 31 edges packed, up to push_big_deg - 1 by
    a warp, longer ones in chunks of push_chunk edges; lists at each bound, with the smallest values of both."""
    off, dst, w = fan(530_000, [1] * 60 + [31, 32, 33, 64, 127, 128, 129, 255, 256, 257, 400, 513], 9)
    exp_b, exp_s = O.bfs(off, dst, 0), O.sssp(off, dst, w, 0)
    with cg.Graph.from_csr(off, dst, w) as g:
        g.set_tuning({"persist_enter": 0, "cluster_enter": 0, "push_block": block, "push_big_deg": 128,
                      "push_chunk": 256})
        np.testing.assert_array_equal(g.run(BFS, 0, cg.make_options(schedule=2, variant=3))[0], exp_b)
        for alpha in (0, 1024):  # every round pushed, every round dense
            g.set_tuning({"sssp_dense_alpha": alpha, "persist_enter": 0, "cluster_enter": 0, "push_block": block,
                          "push_big_deg": 128, "push_chunk": 256})
            np.testing.assert_array_equal(g.run(SSSP, 0, cg.make_options(sssp_delta=1 << 20))[0], exp_s)
        np.testing.assert_array_equal(g.run_batch(BFS, [0, 5])[0][0], exp_b)
