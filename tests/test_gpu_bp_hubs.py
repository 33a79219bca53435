"""Bit-parallel rows of graphs whose hubs' degrees lie around the least degree a
block works on, in degree order and in a random one (where the degrees at the
sampled ids say little), below and above one vertex per block of the grid.
Rows and labels equal the oracle's."""
import numpy as np
import pytest

from helpers import assert_same_unw
from oracle import orc
from parallel_distance_oracle_gb300 import graphs as G

pytestmark = pytest.mark.gpu


def hubs(n, degrees, rng):
    """Hubs of the given degrees over a sparse random graph."""
    u, v = [rng.integers(0, n, n)], [rng.integers(0, n, n)]
    for h, k in enumerate(degrees):
        u.append(np.full(k, h))
        v.append(rng.choice(np.arange(len(degrees), n), k, replace=False))
    u, v = np.concatenate(u), np.concatenate(v)
    key = np.unique(np.minimum(u, v)[u != v] * n + np.maximum(u, v)[u != v])
    return G.csr_from_edges(n, key // n, key % n)


@pytest.mark.parametrize("n,degrees", [(400, [30, 31, 32, 62, 63, 64, 65, 96, 300]), (609, [60, 61, 62, 255, 256, 600]),
                                       (6000, [63, 64, 257, 2046, 2048, 2050, 5900])])
@pytest.mark.parametrize("order", ["degree", "random"])
def test_hub_degrees(cuda_ok, n, degrees, order):
    from parallel_distance_oracle_gb300 import pado
    rng = np.random.Generator(np.random.PCG64(n))
    g = hubs(n, degrees, rng)
    rank = G.degree_rank(g) if order == "degree" else rng.permutation(n).astype(np.uint32)
    got = pado.VertexCentricPLL(g, rank, bp_roots=40, batch=256).export()
    assert_same_unw(got, orc.unw_label(g, rank, 40, 256), order)
