"""Calls that the library refuses with a status, without reading outside their
arrays; the device labels as before afterwards."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import orc
from parallel_distance_oracle_gb300 import graphs as G

pytestmark = pytest.mark.gpu

E_ARG = 1


def _build_ranked(off, adj, w):
    from parallel_distance_oracle_gb300 import _lib as L
    h = C.c_void_p()
    n = len(off) - 1
    off, adj = np.ascontiguousarray(off, np.uint64), np.ascontiguousarray(adj, np.uint32)
    if w is None:
        st = L.lib.pado_unw_build_ranked(n, L.ptr(off), L.ptr(adj), 2, 32, C.byref(h))
    else:
        st = L.lib.pado_w_build_ranked(n, L.ptr(off), L.ptr(adj), L.ptr(np.ascontiguousarray(w, np.uint8)), 32,
                                       C.byref(h))
    return st, h


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("off,first", [
    ([0, 11, 4, 6], 0xFFFFFFFF),  # the first list ends beyond the entries: entry 0 starts no list
    ([0, 11, 4, 6], 2),
    ([0, 5, 3, 6], 2),            # decreasing
    ([0, 2**63, 4, 6], 0xFFFFFFFF),
    ([0, 3, 5, 6], 0xFFFFFFFF),   # well-formed offsets, ids out of range
    ([0, 3, 5, 6], 3),
])
def test_malformed_csr(cuda_ok, weighted, off, first):
    from parallel_distance_oracle_gb300 import _lib as L
    from parallel_distance_oracle_gb300 import pado
    adj = np.array([first, 2, 1, 0, 0, 0], np.uint32)
    st, h = _build_ranked(off, adj, np.full(6, 7, np.uint8) if weighted else None)
    assert st == E_ARG, L.lib.pado_last_error()
    assert not h.value
    g = G.rmat(9, 6, 12, weights=(1, 9))
    rank = G.degree_rank(g)
    got, ref = pado.WeightedVertexCentricPLL(g, rank, batch=64).export(), orc.w_label(g, rank, 64)
    assert np.array_equal(got.off, ref.off) and np.array_equal(got.hub, ref.hub)
