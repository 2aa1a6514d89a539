"""Components of a directed graph without the weak flag (labels pushed along out-edges): lists at the bounds of the
chunks and of the CTAs that take them."""
import numpy as np
import pytest

import cggraph_b200 as cg
from oracle import oracle as O

CC = int(cg.Algorithm_type.CC)


def lists(degrees, V, seed):
    """Vertex i has degrees[i % len(degrees)] random out-neighbours; a chain down from the top carries small labels back."""
    rng = np.random.default_rng(seed)
    deg = np.array([degrees[i % len(degrees)] for i in range(V)])
    src = np.concatenate([np.repeat(np.arange(V), deg), np.arange(0, V - 1, 3)])
    dst = np.concatenate([rng.integers(0, V, int(deg.sum())), np.arange(1, V, 3)])
    key = np.unique(src[src != dst].astype(np.int64) * V + dst[src != dst])
    src, dst = key // V, (key % V).astype(np.uint32)
    off = np.zeros(V + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(src, minlength=V))
    return off, dst


@pytest.mark.gpu
@pytest.mark.parametrize("V,degrees", [
    (2_000, [0, 1, 31, 32, 33, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025]),  # every list of 32 edges in chunks
    (600_000, [0] * 200 + [1, 3] * 20 + [127, 128, 129, 700]),                    # more than 2^19 vertices: by size
    (40_000, [0] * 39_999 + [39_000]),
])
@pytest.mark.parametrize("tuning", [{"push_block": 128}, {"push_block": 256}, {"push_block": 512},
                                    {"push_big_deg": 128, "push_chunk": 256}])
def test_directed_components(V, degrees, tuning):
    off, dst = lists(degrees, V, seed=V)
    exp = O.cc(off, dst)
    with cg.Graph.from_csr(off, dst) as g:
        g.set_tuning(tuning)
        np.testing.assert_array_equal(g.run(CC, 0)[0], exp)
        assert g.stats().cc_path == 1
