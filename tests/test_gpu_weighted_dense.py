"""Weighted labeling of graphs in which thousands of vertices have long lists:
only as many as WHEAVY_MAX (8,192) of them are split over the grid."""
import numpy as np
import pytest

from helpers import assert_same_w
from oracle import orc
from parallel_distance_oracle_gb300 import graphs as G

pytestmark = pytest.mark.gpu


def repeated_tree(n, copies, seed):
    """A binary tree with every edge `copies` times, each with a weight of its own:
    lists of `copies` entries and more, and few labels."""
    rng = np.random.Generator(np.random.PCG64(seed))
    v = np.repeat(np.arange(1, n), copies)
    u = (v - 1) // 2
    w = rng.integers(1, 101, len(v))
    src, dst, ww = np.concatenate([u, v]), np.concatenate([v, u]), np.concatenate([w, w])
    o = np.lexsort((dst, src))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(src, minlength=n))
    return G.CSRGraph(n, off, dst[o].astype(np.uint32), ww[o].astype(np.uint8))


# all lists have 512 entries or more, at the limit and beyond it (where those of 1,024 are
# split); half of them; all have 1,024 or more
@pytest.mark.parametrize("n,copies,B", [(8192, 512, 512), (8193, 512, 128), (9001, 511, 64), (8200, 1024, 512)])
def test_limit(cuda_ok, n, copies, B):
    from parallel_distance_oracle_gb300 import pado
    g = repeated_tree(n, copies, n)
    # by level of the tree, in any order within one
    rank = np.empty(n, np.uint32)
    rank[np.lexsort((np.random.Generator(np.random.PCG64(copies)).random(n), np.log2(np.arange(n) + 1).astype(int)))] = \
        np.arange(n)
    got = pado.WeightedVertexCentricPLL(g, rank, batch=B).export()
    assert_same_w(got, orc.w_label(g, rank, B))


def test_time_of_small_batches(cuda_ok):
    """12,000 vertices of average degree 800: four times the batches took 1.1 times
    as long before lists were split, 1.7 times with all of them split."""
    from parallel_distance_oracle_gb300 import pado
    n, rng = 12000, np.random.Generator(np.random.PCG64(1))
    m = n * 400
    g = G.csr_from_edges(n, rng.integers(0, n, m), rng.integers(0, n, m), rng.integers(1, 101, m))
    rank = G.degree_rank(g)

    def best(B):
        t = []
        for _ in range(3):
            x = pado.WeightedVertexCentricPLL(g, rank, batch=B)
            t.append(x.info().build_seconds)
            x.close()
        return min(t)

    assert best(128) < 1.45 * best(512)
