"""Unweighted labeling of graphs without hubs, whose label loop takes a lane per
candidate in the second bit-parallel stage and covers candidates a batch at a
time in the distance test: root counts around the 16-byte rows of BP distances,
batch sizes around the words of a batch's bitmaps, distances beyond them (long
grids), alone and as a union.  Labels equal the oracle's."""
import numpy as np
import pytest

from helpers import assert_same_unw
from oracle import orc
from parallel_distance_oracle_gb300 import graphs as G

pytestmark = pytest.mark.gpu


def long_grid(n, rows=6):
    """A strip of `rows` rows: distances far beyond a random graph's."""
    i = np.arange(n)
    right, down = i[i + rows < n], i[(i % rows != rows - 1) & (i + 1 < n)]
    return G.csr_from_edges(n, np.concatenate([right, down]), np.concatenate([right + rows, down + 1]))


def check(g, K, B, rank=None):
    from parallel_distance_oracle_gb300 import pado
    rank = G.degree_rank(g) if rank is None else rank
    got = pado.VertexCentricPLL(g, rank, bp_roots=K, batch=B).export()
    assert_same_unw(got, orc.unw_label(g, rank, K, B), f"K={K} B={B}")


@pytest.mark.parametrize("K", [0, 1, 2, 15, 16, 17, 31, 32, 33, 48, 50, 63, 64])
def test_root_counts(cuda_ok, K):
    check(G.erdos_renyi(1500, 6, 200 + K), K, 256)


@pytest.mark.parametrize("B", [1, 32, 33, 96, 127, 128, 129, 256, 384, 500, 512, 1000, 1024, 2000, 2048])
def test_batch_sizes(cuda_ok, B):
    check(G.erdos_renyi(2300, 5, 300 + B), 8, B)


@pytest.mark.parametrize("rows,B", [(2, 128), (3, 256), (6, 512), (20, 1024)])
def test_long_distances(cuda_ok, rows, B):
    n = min(rows * 200, 2400)
    rng = np.random.Generator(np.random.PCG64(rows))
    check(long_grid(n, rows), 4, B, rng.permutation(n).astype(np.uint32))


def test_union(cuda_ok):
    from parallel_distance_oracle_gb300 import pado
    gs = [G.erdos_renyi(1200, 6, 41), long_grid(900, 5), G.grid_with_shortcuts(1600, 0.02, 42), G.erdos_renyi(300, 4, 43)]
    rks = [G.degree_rank(g) for g in gs]
    for idx, g, rk in zip(pado.build_many(gs, rks, bp_roots=20, batch=128), gs, rks):
        assert_same_unw(idx.export(), orc.unw_label(g, rk, 20, 128))


def test_growing_pool(cuda_ok, monkeypatch):
    """Levels re-run after the label pool grows."""
    monkeypatch.setenv("PADO_DEBUG_POOL_ENTRIES", "4096")
    check(G.erdos_renyi(1800, 6, 77), 16, 256)
