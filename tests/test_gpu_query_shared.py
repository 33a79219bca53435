"""Queries on label lists that share all their hubs, or none, over several
windows: batches of one pair per warp, which read ahead, and of groups."""
import numpy as np
import pytest

from oracle import orc

pytestmark = pytest.mark.gpu

N = 650


def _lists(kind):
    """Vertex v's list: every hub up to v, or every other one (even for even v)."""
    hubs = [np.arange(v + 1) if kind == "all" else np.arange(v % 2, v + 1, 2) for v in range(N)]
    off = np.zeros(N + 1, np.uint64)
    off[1:] = np.cumsum([len(h) for h in hubs])
    return off, np.concatenate(hubs).astype(np.uint32)


@pytest.mark.parametrize("k", [1, 1000, 77_823, 200_003])
@pytest.mark.parametrize("kind", ["all", "half"])
@pytest.mark.parametrize("weighted", [False, True])
def test_shared_hubs(cuda_ok, weighted, kind, k):
    from parallel_distance_oracle_gb300 import pado
    rng = np.random.Generator(np.random.PCG64(k))
    off, hub = _lists(kind)
    a, b = rng.integers(0, N, (2, k)).astype(np.uint32)
    a[:1], b[:1] = N - 1, N - 3
    if weighted:
        dist = rng.integers(0, 32767, len(hub)).astype(np.int16)
        idx = pado.WeightedVertexCentricPLL.from_labels(pado.CanonicalLabels(N, 0, off, hub, dist))
        want = orc.w_query(orc.WLabels(N, off, hub, dist), a, b)
    else:
        dist = rng.integers(100, 255, len(hub)).astype(np.uint8)
        idx = pado.VertexCentricPLL.from_labels(pado.CanonicalLabels(N, 0, off, hub, dist))
        want = orc.unw_query(orc.UnwLabels(N, 0, off, hub, dist, np.zeros(1), np.zeros(2)), a, b)
    assert np.array_equal(idx.query(a, b), want)
