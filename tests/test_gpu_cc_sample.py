"""Components where the sampled link rounds find one giant tree, many equal ones, or none."""
import numpy as np
import pytest

import cggraph_b200 as cg
from oracle import oracle as O

CC = int(cg.Algorithm_type.CC)
WEAK = 0x8


def blocks(sizes, extra, seed):
    """Disjoint random trees of the given sizes over shuffled ids (parents skewed to a hub), plus `extra` lone vertices."""
    rng = np.random.default_rng(seed)
    V = int(sum(sizes)) + extra
    ids = rng.permutation(V)
    src, dst, base = [], [], 0
    for n in sizes:
        child = np.arange(1, n)
        parent = np.where(rng.random(n - 1) < 0.5, 0, (rng.random(n - 1) * child).astype(np.int64))
        a, b = ids[base + child], ids[base + parent]
        flip = rng.random(n - 1) < 0.5  # edges point either way
        src.append(np.where(flip, a, b))
        dst.append(np.where(flip, b, a))
        base += n
    return V, np.concatenate(src), np.concatenate(dst)


def csr(V, src, dst):
    key = np.unique(src.astype(np.int64) * V + dst)
    src, dst = key // V, (key % V).astype(np.uint32)
    off = np.zeros(V + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(src, minlength=V))
    return off, dst


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,extra", [
    ([200_000, 3, 2], 5_000),
    ([300] * 400, 1),
    ([130, 2, 2, 2], 0),            # fewer vertices than one sample step
    ([70_000, 70_000, 70_001], 33),
    ([5_000_000, 1_000], 100_000),  # rounds above 2^22 vertices
])
def test_components(sizes, extra):
    V, src, dst = blocks(sizes, extra, seed=len(sizes) + extra)
    off, dd = csr(V, src, dst)
    soff, sdst = csr(V, np.concatenate([src, dst]), np.concatenate([dst, src]))
    exp = O.cc(soff, sdst)
    with cg.Graph.from_csr(off, dd) as g:
        np.testing.assert_array_equal(g.run(CC, 0, cg.make_options(flags=WEAK))[0], exp)
    with cg.Graph.from_csr(soff, sdst) as g:
        np.testing.assert_array_equal(g.run(CC, 0)[0], exp)


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,degree", [
    ([1 << 18], 8),                    # one component, no vertex of 64 edges
    ([40_000, 40_000, 17, 5], 4),
    ([12] * 9_000, 7),                 # none that a sample would find often
    ([1 << 18], 1),                    # trees and cycles
    ([4_300_000], 3),                  # rounds above 2^22 vertices
])
def test_components_without_hubs(sizes, degree):
    rng = np.random.default_rng(len(sizes) + degree)
    V = sum(sizes) + 3
    base = np.concatenate([[0], np.cumsum(sizes)])
    ids = rng.permutation(V)
    src = np.concatenate([np.repeat(np.arange(b, b + n), degree) for b, n in zip(base, sizes)])
    dst = np.concatenate([b + rng.integers(0, n, n * degree) for b, n in zip(base, sizes)])
    keep = src != dst
    src, dst = ids[src[keep]], ids[dst[keep]]
    off, dd = csr(V, src, dst)
    soff, sdst = csr(V, np.concatenate([src, dst]), np.concatenate([dst, src]))
    longest = int(np.diff(soff.astype(np.int64)).max())
    assert longest < 64
    exp = O.cc(soff, sdst)
    with cg.Graph.from_csr(off, dd) as g:
        np.testing.assert_array_equal(g.run(CC, 0, cg.make_options(flags=WEAK))[0], exp)
    with cg.Graph.from_csr(soff, sdst) as g:
        np.testing.assert_array_equal(g.run(CC, 0)[0], exp)


@pytest.mark.gpu
@pytest.mark.parametrize("V", [(1 << 14) - 1, 1 << 14, (1 << 14) + 1])
def test_components_at_the_smallest_sampled_graph(V):
    for hub in (0, 200):
        rng = np.random.default_rng(V + hub)
        src = np.concatenate([rng.integers(0, V, 2 * V), np.zeros(hub, np.int64)])
        dst = np.concatenate([rng.integers(0, V, 2 * V), rng.integers(0, V, hub)])
        keep = src != dst
        off, dd = csr(V, src[keep], dst[keep])
        soff, sdst = csr(V, np.concatenate([src[keep], dst[keep]]), np.concatenate([dst[keep], src[keep]]))
        exp, launches = O.cc(soff, sdst), []
        with cg.Graph.from_csr(off, dd) as g:
            np.testing.assert_array_equal(g.run(CC, 0, cg.make_options(flags=WEAK))[0], exp)
            launches.append(g.stats().launches)
        if hub:
            assert launches[0] == (8 if V < 1 << 14 else 11)
        with cg.Graph.from_csr(soff, sdst) as g:
            np.testing.assert_array_equal(g.run(CC, 0)[0], exp)
