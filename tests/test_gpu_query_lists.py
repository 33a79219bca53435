"""Query kernels on label lists of chosen lengths: around the 32-hub groups of
the shorter list and the windows of the longer one, with disjoint, interleaved
and equal hub ranges, and bit-parallel rows whose distance sums cover the
skipped (below 2, above 257) and tied cases.  Integers, equal to the oracle."""
import numpy as np
import pytest

from oracle import orc
from parallel_distance_oracle_gb300 import graphs as G

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 31, 32, 33, 64, 127, 128, 129, 160, 255, 256, 257, 384, 700]


def label_lists(rng, n):
    """Vertex i has LENGTHS[i % len] hubs: spread over all ids, packed low, or
    packed high by turns."""
    off, hubs = [0], []
    for i in range(n):
        k = LENGTHS[i % len(LENGTHS)]
        lo, hi = [(0, n), (0, max(k, n // 3)), (n - max(k, n // 3), n)][i // len(LENGTHS) % 3]
        hubs.append(np.sort(rng.choice(np.arange(lo, hi), k, replace=False)))
        off.append(off[-1] + k)
    return np.array(off, np.uint64), np.concatenate(hubs).astype(np.uint32)


def all_pairs(rng, n):
    a, b = np.meshgrid(np.arange(3 * len(LENGTHS)), np.arange(3 * len(LENGTHS)))
    r = rng.integers(0, n + 2, (2, 3000))  # ids n and n + 1 are out of range
    return np.concatenate([a.ravel(), r[0]]).astype(np.uint32), np.concatenate([b.ravel(), r[1]]).astype(np.uint32)


@pytest.mark.parametrize("K", [0, 1, 31, 33, 64])
def test_unweighted_lists(cuda_ok, K):
    from parallel_distance_oracle_gb300 import pado
    rng = np.random.Generator(np.random.PCG64(100 + K))
    n = 1500
    off, hub = label_lists(rng, n)
    dist = rng.integers(0, 250, len(hub)).astype(np.uint8)
    bpd = rng.choice(np.array([0, 1, 2, 3, 4, 120, 127, 128, 129, 130, 255], np.uint8), n * K)
    if K:
        bpd.reshape(n, K)[::7] = 255  # vertices that no root reaches
    bps = np.where(rng.random(2 * n * K) < 0.6, 0, 1 << rng.integers(0, 4, 2 * n * K)).astype(np.uint64)
    lab = orc.UnwLabels(n, K, off, hub, dist, bpd, bps)
    a, b = all_pairs(rng, n)
    idx = pado.VertexCentricPLL.from_labels(pado.CanonicalLabels(n, K, off, hub, dist, bpd, bps))
    assert np.array_equal(idx.query(a, b), orc.unw_query(lab, a, b))


def test_weighted_lists(cuda_ok):
    from parallel_distance_oracle_gb300 import pado
    rng = np.random.Generator(np.random.PCG64(7))
    n = 1500
    off, hub = label_lists(rng, n)
    dist = rng.integers(0, 32767, len(hub)).astype(np.int16)
    a, b = all_pairs(rng, n)
    idx = pado.WeightedVertexCentricPLL.from_labels(pado.CanonicalLabels(n, 0, off, hub, dist))
    assert np.array_equal(idx.query(a, b), orc.w_query(orc.WLabels(n, off, hub, dist), a, b))


def test_served_lists(cuda_ok):
    from parallel_distance_oracle_gb300 import pado
    g = G.erdos_renyi(4000, 8, 11)  # lists of up to hundreds of labels
    rk = G.degree_rank(g)
    idx = pado.VertexCentricPLL(g, rk, bp_roots=2, batch=512)
    a, b = G.random_pairs(g.n, 20011, 5)
    want = idx.query(a, b)
    srv = pado.Server(1 << 30, max_batch_pairs=4096)
    i = srv.add(idx)
    assert np.array_equal(srv.query(i, a, b), want)
    srv.close()
