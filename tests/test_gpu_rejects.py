"""Calls with arguments that are not what the library asks for: refused with a
status, or answered, without an access outside their arrays; the library works as
before afterwards."""
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


@pytest.mark.parametrize("k", [1, 300, 20000])
@pytest.mark.parametrize("which", ["a", "b", "out"])
def test_query_with_a_device_array(cuda_ok, which, k):
    """pado_query takes host arrays.  A device array in the place of one goes
    through the runtime's copies: a status or the right distances, and the host
    never touches it."""
    import torch

    from parallel_distance_oracle_gb300 import _lib as L
    from parallel_distance_oracle_gb300 import pado
    g = G.rmat(9, 6, 12)
    idx = pado.VertexCentricPLL(g, G.degree_rank(g), bp_roots=8, batch=64)
    rng = np.random.Generator(np.random.PCG64(k))
    a, b = (rng.integers(0, g.n, k).astype(np.uint32) for _ in range(2))
    ref, out = idx.query(a, b), np.zeros(k, np.uint8)
    host = {"a": a.view(np.int32), "b": b.view(np.int32), "out": out}
    dev = torch.from_numpy(host[which]).cuda()
    torch.cuda.synchronize()
    p = {x: L.ptr(y) for x, y in host.items()} | {which: C.c_void_p(dev.data_ptr())}
    st = L.lib.pado_query(idx._need(), k, p["a"], p["b"], p["out"])
    assert st != 0 or np.array_equal(dev.cpu().numpy() if which == "out" else out, ref)
    # the caller's own arrays are untouched and ordinary calls go on
    assert np.array_equal(idx.query(a, b), ref)
