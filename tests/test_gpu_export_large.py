"""Exports in original-id order of more than 32 MiB, which the gather kernel writes
into page-locked destinations itself while others go through device buffers: every
mix of the two against the arrays the index came from."""

import ctypes as C

import numpy as np
import pytest
import torch

from parallel_distance_oracle_gb300 import _lib, pado
from parallel_distance_oracle_gb300.pado import CanonicalLabels

pytestmark = pytest.mark.gpu

STAGED = 32 << 20  # up to here an export is gathered into device scratch


def _labels(n, K, most, weighted):
    rng = np.random.default_rng(n + K)
    cnt = rng.integers(0, most + 1, n)
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(cnt)
    hubs = np.cumsum(rng.integers(1, n // most, (n, most)), axis=1)  # ascending, below n
    hub = hubs[np.arange(most) < cnt[:, None]].astype(np.uint32)
    dist = rng.integers(0, 200, len(hub)).astype(np.int16 if weighted else np.uint8)
    bpd = rng.integers(0, 255, n * K).astype(np.uint8) if K else None
    bps = rng.integers(0, 1 << 63, 2 * n * K).astype(np.uint64) if K else None
    return CanonicalLabels(n, K, off, hub, dist, bpd, bps)


@pytest.mark.parametrize("pinned", ["all", "even", "odd", "none"])
@pytest.mark.parametrize("n,K,most,weighted", [(40_003, 50, 20, False), (30_011, 0, 400, True), (16_001, 64, 600, False)])
def test_mixes(n, K, most, weighted, pinned):
    ref = _labels(n, K, most, weighted)
    rank = np.random.default_rng(3).permutation(n).astype(np.uint32)
    b, e = ref.off[rank].astype(np.int64), ref.off[rank.astype(np.int64) + 1].astype(np.int64)
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(e - b)
    pick = np.repeat(b - off[:-1].astype(np.int64), e - b) + np.arange(int(off[-1]))
    want = [off, ref.hub[pick], ref.dist[pick]]
    if K:
        want += [ref.bpd.reshape(n, K)[rank], ref.bps.reshape(n, 2 * K)[rank]]
    assert sum(x.nbytes for x in want) > STAGED

    index = (pado.WeightedVertexCentricPLL if weighted else pado.VertexCentricPLL).from_labels(ref)
    index.order_labels(rank=rank)
    lock = {"all": lambda i: True, "even": lambda i: i % 2 == 0, "odd": lambda i: i % 2 == 1, "none": lambda i: False}
    bufs = [torch.full((x.nbytes + 64,), 0xEE, dtype=torch.uint8, pin_memory=lock[pinned](i))
            for i, x in enumerate(want)]
    # 16 bytes past each start, a guard on both sides
    ptrs = [C.c_void_p(t.data_ptr() + 16) for t in bufs] + ([] if K else [None, None])
    _lib.check(_lib.lib.pado_export(index._need(), *ptrs))
    for x, t in zip(want, bufs):
        a = t.numpy()
        assert (a[:16] == 0xEE).all() and (a[16 + x.nbytes:] == 0xEE).all()
        assert a[16:16 + x.nbytes].tobytes() == np.ascontiguousarray(x).tobytes()
    index.close()
