"""Device memory of a build.  The label pool that it starts with on graphs without
hubs: larger than with hubs, but bounded, and a build that cannot have it (or what
else its variant of the loop allocates) goes on with what a graph with hubs gets.
Tables that only one variant reads are that variant's."""
from __future__ import annotations

import ctypes as C
import threading
import time

import numpy as np
import pytest

from helpers import assert_same_unw
from oracle import orc
from parallel_distance_oracle_gb300 import graphs as G

pytestmark = pytest.mark.gpu

E_NOMEM = 2


def _peak(build):
    """Device bytes held at most during build(), run three times after a first one
    (which loads the library's kernels)."""
    import torch
    build()
    torch.cuda.synchronize()
    free0 = least = torch.cuda.mem_get_info()[0]
    done = threading.Event()

    def watch():
        nonlocal least
        while not done.is_set():
            least = min(least, torch.cuda.mem_get_info()[0])
            time.sleep(0.0005)

    t = threading.Thread(target=watch)
    t.start()
    try:
        for _ in range(3):
            build()
    finally:
        done.set()
        t.join()
    return free0 - least


def test_memory_of_a_tree(cuda_ok):
    """A binary tree of 524,287 vertices has a dozen labels per vertex; a build that
    starts with 256 pool entries per vertex holds 2.4 GB."""
    from parallel_distance_oracle_gb300 import pado
    n = (1 << 19) - 1
    v = np.arange(1, n)
    g = G.csr_from_edges(n, (v - 1) // 2, v)
    rank = np.arange(n, dtype=np.uint32)
    assert _peak(lambda: pado.VertexCentricPLL(g, rank, bp_roots=64, batch=1024).close()) < 4e9


def test_memory_of_padded_rows(cuda_ok):
    """With hubs nothing reads the 16-byte rows of BP distances: K = 50 holds two
    roots' rows (34 bytes a vertex) more than K = 48, not 64 bytes on top."""
    from parallel_distance_oracle_gb300 import pado
    n = 1 << 21
    g = G.csr_from_edges(n, np.zeros(n - 1, np.int64), np.arange(1, n))
    rank = np.arange(n, dtype=np.uint32)
    peak = [_peak(lambda: pado.VertexCentricPLL(g, rank, bp_roots=K, batch=1024).close()) for K in (48, 50)]
    assert peak[1] - peak[0] < (34 + 16) * n


def _build(L, g, rank, K, B):
    h = C.c_void_p()
    st = L.lib.pado_unw_build(g.n, L.ptr(np.ascontiguousarray(g.off, np.uint64)),
                              L.ptr(np.ascontiguousarray(g.adj, np.uint32)), L.ptr(rank), K, B, C.byref(h))
    return st, h


def test_failed_allocation_without_hubs(cuda_ok):
    """One allocation of a build fails, each in turn.  A graph with hubs gets
    PADO_E_NOMEM for all of them; one without gets its labels when the failure
    comes in the labeling, and nothing stays allocated either way."""
    from parallel_distance_oracle_gb300 import _lib as L
    from parallel_distance_oracle_gb300 import pado
    K, B = 8, 128
    live = L.lib.pado_debug_live_allocations()

    def statuses(g, rank, upto):
        out = []
        ref = orc.unw_label(g, rank, K, B)
        for n in range(1, upto + 1):
            L.lib.pado_debug_fail_alloc(n)
            st, h = _build(L, g, rank, K, B)
            L.lib.pado_debug_fail_alloc(0)
            assert st in (0, E_NOMEM), (n, L.lib.pado_last_error())
            if st == 0:
                x = pado.VertexCentricPLL()
                x._h = h
                assert_same_unw(x.export(), ref, f"allocation {n}")
                x.close()
            assert L.lib.pado_debug_live_allocations() == live, n
            out.append(st)
        return out

    hub_g, flat_g = G.rmat(10, 8, 5), G.erdos_renyi(1024, 6, 6)
    hub_r, flat_r = (G.degree_rank(g).astype(np.uint32) for g in (hub_g, flat_g))
    hub = statuses(hub_g, hub_r, 40)
    flat = statuses(flat_g, flat_r, 40)
    assert 5 < hub.count(E_NOMEM) < 40
    assert flat.count(E_NOMEM) < hub.count(E_NOMEM) - 3
    # the failures before the labeling still end the build, those in it no longer
    first_ok = flat.index(0)
    assert all(s == E_NOMEM for s in flat[:first_ok])
