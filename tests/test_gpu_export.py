"""Exports in original-id order against the arrays they came from: sizes around
a step of the offsets' scan and both sides of its limit, and destinations of
every alignment in page-locked and pageable memory."""

import ctypes as C

import numpy as np
import pytest
import torch

from parallel_distance_oracle_gb300 import _lib, pado
from parallel_distance_oracle_gb300.pado import CanonicalLabels

pytestmark = pytest.mark.gpu


def _labels(rng, n, K, weighted):
    cnt = rng.integers(0, min(n, 9) + 1, n)
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(cnt)
    hub = np.concatenate([np.sort(rng.choice(n, c, replace=False)) for c in cnt] + [[]]).astype(np.uint32)
    dist = rng.integers(0, 200, len(hub)).astype(np.int16 if weighted else np.uint8)
    bpd = rng.integers(0, 255, n * K).astype(np.uint8) if K else None
    bps = rng.integers(0, 1 << 63, 2 * n * K).astype(np.uint64) if K else None
    return CanonicalLabels(n, K, off, hub, dist, bpd, bps)


@pytest.mark.parametrize("n,K,weighted,shift,pinned", [
    (1, 3, False, 0, True), (33, 50, False, 1, True), (4095, 0, True, 2, True), (4096, 5, False, 3, True),
    (4097, 16, False, 7, False), (8191, 1, False, 13, True), (16384, 2, False, 4, True), (16385, 0, True, 8, True),
    (16385, 3, False, 15, True)])
def test_export_in_original_order(n, K, weighted, shift, pinned):
    rng = np.random.default_rng(n + shift)
    ref = _labels(rng, n, K, weighted)
    rank = rng.permutation(n).astype(np.uint32)
    cls = pado.WeightedVertexCentricPLL if weighted else pado.VertexCentricPLL
    index = cls.from_labels(ref)
    index.order_labels(rank=rank)
    tot = len(ref.hub)
    dsz = ref.dist.itemsize

    def room(nbytes, unit):
        # `shift` units past a page-locked or pageable start, a guard at the end
        t = torch.full((nbytes + (shift + 1) * unit + 16,), 0xEE, dtype=torch.uint8, pin_memory=pinned)
        return t, t.data_ptr() + shift * unit

    sizes = [((n + 1) * 8, 8), (tot * 4, 4), (tot * dsz, dsz)] + ([(n * K, 1), (n * K * 16, 8)] if K else [])
    bufs = [room(*x) for x in sizes]
    ptrs = [C.c_void_p(p) for _, p in bufs] + ([] if K else [None, None])
    _lib.check(_lib.lib.pado_export(index._need(), *ptrs))
    got = []
    for (nbytes, unit), (t, _) in zip(sizes, bufs):
        a = t.numpy()
        assert (a[:shift * unit] == 0xEE).all() and (a[shift * unit + nbytes:] == 0xEE).all()
        got.append(a[shift * unit:shift * unit + nbytes].tobytes())

    b, e = ref.off[rank].astype(np.int64), ref.off[rank.astype(np.int64) + 1].astype(np.int64)
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(e - b)
    pick = np.concatenate([np.arange(x, y) for x, y in zip(b, e)] + [[]]).astype(np.int64)
    want = [off, ref.hub[pick], ref.dist[pick]]
    if K:
        want += [ref.bpd.reshape(n, K)[rank], ref.bps.reshape(n, 2 * K)[rank]]
    for w, g in zip(want, got):
        assert np.ascontiguousarray(w).tobytes() == g
    index.close()
