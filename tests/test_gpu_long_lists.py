"""Unweighted labeling whose distance tests walk long label lists: a spider of m
legs of two vertices, ranked inner vertices first, then outer ones, the centre
last.  An outer vertex holds a label to every inner one, and at level 4 the root
r' of another leg is covered by exactly one of them -- at its own place in the
list, so that candidates leave in every staged window of the block path (1,024
entries, the last batches) and the warp path (384).  Labels equal the oracle's."""
import numpy as np
import pytest

from helpers import assert_same_unw
from oracle import orc
from parallel_distance_oracle_gb300 import graphs as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("legs,batch", [(380, 512), (390, 96), (1020, 64), (1030, 64), (1300, 128)])
def test_spider(cuda_ok, legs, batch):
    from parallel_distance_oracle_gb300 import pado
    i = np.arange(legs)
    n = 2 * legs + 1
    g = G.csr_from_edges(n, np.concatenate([i, i]), np.concatenate([legs + i, np.full(legs, n - 1)]))
    rng = np.random.Generator(np.random.PCG64(legs))
    rank = np.concatenate([rng.permutation(legs), legs + rng.permutation(legs), [n - 1]]).astype(np.uint32)
    got = pado.VertexCentricPLL(g, rank, bp_roots=0, batch=batch).export()
    assert_same_unw(got, orc.unw_label(g, rank, 0, batch))
