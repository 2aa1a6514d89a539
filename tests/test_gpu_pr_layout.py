"""PageRank rows at the bounds of the layout: long rows, their segments, hub rows."""
import numpy as np
import pytest

import cggraph_b200 as cg
from oracle import oracle as O

PR = int(cg.Algorithm_type.PR)


def rows_graph(V, in_degrees, extra, seed):
    """Vertex i has in_degrees[i] in-edges from random others; `extra` more random edges."""
    rng = np.random.default_rng(seed)
    src, dst = [], []
    for i, d in enumerate(in_degrees):
        s = rng.choice(V - 1, size=d, replace=False)
        src.append(s + (s >= i))
        dst.append(np.full(d, i))
    s, t = rng.integers(0, V, extra), rng.integers(len(in_degrees), V, extra)
    src, dst = np.concatenate(src + [s]), np.concatenate(dst + [t])
    key = np.unique(src[src != dst].astype(np.int64) * V + dst[src != dst])
    src, dst = key // V, (key % V).astype(np.uint32)
    off = np.zeros(V + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(src, minlength=V))
    return off, dst


# edges below 2^22: rows of 64 or more are cut into segments of at most 32,
# more than 128 segments make a hub row; above, 128 and 64
@pytest.mark.gpu
@pytest.mark.parametrize("V,degrees,extra", [
    (9000, [0, 1, 31, 32, 33, 63, 64, 65, 96, 97, 127, 4095, 4096, 4097, 4128, 8191], 500),
    (33, [0, 32, 31], 40),
    (300_000, [63, 64, 127, 128, 129, 191, 192, 193, 8191, 8192, 8193, 8256, 200_000], 4_400_000),
])
@pytest.mark.parametrize("iters", [1, 2, 7])
def test_row_bounds(V, degrees, extra, iters):
    off, dst = rows_graph(V, degrees, extra, seed=V + len(degrees))
    exp = O.pagerank(off, dst, iters)
    with cg.Graph.from_csr(off, dst) as g:
        got, _ = g.run(PR, iters)
        again, _ = g.run(PR, iters)
    # a sum of at most V terms, all positive: relative error below V * 2^-53 per iteration on either side
    np.testing.assert_allclose(got, exp, rtol=2 * iters * V * 2.0 ** -53 + 1e-14, atol=0)
    np.testing.assert_array_equal(got, again)


@pytest.mark.gpu
@pytest.mark.parametrize("V,degree,hub", [(5, 1, 0), (4_096, 8, 0), (131_072, 30, 0), (100_000, 3, 90_000)])
def test_overlapped_iterations(V, degree, hub):
    """Each iteration's kernels are placed while those before them run: many iterations of graphs that fit the machine
    at once, with and without long rows, against the oracle and against launches without the overlap."""
    rng = np.random.default_rng(V)
    src = np.concatenate([np.repeat(np.arange(V), degree), 1 + rng.integers(0, V - 1, hub)])
    dst = np.concatenate([rng.integers(0, V, V * degree), np.zeros(hub, np.int64)])
    key = np.unique(src[src != dst].astype(np.int64) * V + dst[src != dst])
    off = np.zeros(V + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(key // V, minlength=V))
    dd = (key % V).astype(np.uint32)
    iters = 60
    exp = O.pagerank(off, dd, iters)
    with cg.Graph.from_csr(off, dd) as g:
        got = [g.run(PR, iters)[0] for _ in range(3)]
        plain, _ = g.run(PR, iters, cg.make_options(flags=0x1))  # timed launches are not overlapped
    np.testing.assert_allclose(plain, exp, rtol=2 * iters * V * 2.0 ** -53 + 1e-14, atol=0)
    for x in got:
        np.testing.assert_array_equal(x, plain)
