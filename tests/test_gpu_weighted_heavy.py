"""Weighted labeling of graphs whose vertices' degrees lie around the heavy-tail
limit (512) and its items (64 entries): the tails whose relaxations the whole grid
gathers and whose checks a block does.  Labels equal the oracle's; also when the
round log starts tiny, so that heavy tails are re-run after it grows, and under
the host-driven loop, which has no heavy tails."""
import numpy as np
import pytest

from helpers import assert_same_w
from oracle import orc
from parallel_distance_oracle_gb300 import graphs as G

pytestmark = pytest.mark.gpu

HUB_DEGREES = [511, 512, 513, 575, 576, 577, 900, 1500]


def hub_graph(seed, n=2500):
    rng = np.random.Generator(np.random.PCG64(seed))
    u, v = [rng.integers(0, n, 3 * n)], [rng.integers(0, n, 3 * n)]
    # the hubs take turns as the first ids, so that hubs neighbour hubs
    for h, d in enumerate(HUB_DEGREES):
        u.append(np.full(d, h))
        v.append(rng.choice(np.arange(1, n), d, replace=False))
    u, v = np.concatenate(u), np.concatenate(v)
    return G.csr_from_edges(n, u, v, rng.integers(1, 101, len(u)))


def labels(g, rank, batch):
    from parallel_distance_oracle_gb300 import pado
    idx = pado.WeightedVertexCentricPLL(g, rank, batch=batch)
    out = idx.export()
    idx.close()
    return out


@pytest.mark.parametrize("batch", [4, 64, 512, 1000, 2048])
def test_heavy_tails(cuda_ok, batch, monkeypatch):
    g = hub_graph(batch)
    rank = G.degree_rank(g)
    want = orc.w_label(g, rank, batch)
    assert_same_w(labels(g, rank, batch), want, "persistent loop")
    monkeypatch.setenv("PADO_DEBUG_POOL_ENTRIES", "2048")
    assert_same_w(labels(g, rank, batch), want, "tiny logs and pool")
    monkeypatch.delenv("PADO_DEBUG_POOL_ENTRIES")
    monkeypatch.setenv("PADO_LEVEL_LOOP", "host")
    assert_same_w(labels(g, rank, batch), want, "host-driven loop")


def test_unsorted_ranks(cuda_ok):
    """Heavy vertices late in the order: heavy tails in later batches too."""
    g = hub_graph(3)
    rank = G.degree_rank(g)
    rank = (g.n - 1 - rank.astype(np.int64)).astype(np.uint32)
    assert_same_w(labels(g, rank, 64), orc.w_label(g, rank, 64), "reversed order")
