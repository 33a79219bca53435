"""Query batches at the sizes where a warp's group of pairs changes (1 to 2, 2
to 4, 32), with a remainder in the last group: lists on both sides of 32 hubs,
empty lists and out-of-range ids in one group.  Integers, equal to the oracle."""
import numpy as np
import pytest

from oracle import orc

pytestmark = pytest.mark.gpu

N = 900


def _lists(rng):
    cnt = rng.choice([0, 1, 5, 31, 32, 33, 40], N)
    off = np.zeros(N + 1, np.uint64)
    off[1:] = np.cumsum(cnt)
    return off, np.concatenate([np.sort(rng.choice(N, c, replace=False)) for c in cnt]).astype(np.uint32)


@pytest.mark.parametrize("k", [38912, 77823, 77824, 77841, 155651, 1245184 + 17])
@pytest.mark.parametrize("weighted", [False, True])
def test_query_groups(cuda_ok, k, weighted):
    from parallel_distance_oracle_gb300 import pado
    rng = np.random.Generator(np.random.PCG64(k))
    off, hub = _lists(rng)
    a, b = rng.integers(0, N + 3, (2, k)).astype(np.uint32)  # the last three ids are out of range
    if weighted:
        dist = rng.integers(0, 32767, len(hub)).astype(np.int16)
        idx = pado.WeightedVertexCentricPLL.from_labels(pado.CanonicalLabels(N, 0, off, hub, dist))
        want = orc.w_query(orc.WLabels(N, off, hub, dist), a, b)
    else:
        K = 40
        dist = rng.integers(0, 250, len(hub)).astype(np.uint8)
        bpd = rng.choice(np.array([0, 1, 2, 100, 127, 128, 129, 255], np.uint8), N * K)
        bps = np.where(rng.random(2 * N * K) < 0.6, 0, 1 << rng.integers(0, 4, 2 * N * K)).astype(np.uint64)
        idx = pado.VertexCentricPLL.from_labels(pado.CanonicalLabels(N, K, off, hub, dist, bpd, bps))
        want = orc.unw_query(orc.UnwLabels(N, K, off, hub, dist, bpd, bps), a, b)
    assert np.array_equal(idx.query(a, b), want)
