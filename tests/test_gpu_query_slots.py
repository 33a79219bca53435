"""pado_query from more threads than slots are kept, beside larger queries and
calls that give the kept slots and scratch back."""
import threading

import numpy as np
import pytest

from oracle import orc
from parallel_distance_oracle_gb300 import graphs as G

pytestmark = pytest.mark.gpu


def test_threads(cuda_ok):
    from parallel_distance_oracle_gb300 import _lib, pado
    g = G.rmat(11, 8, 4)
    rank = G.degree_rank(g)
    idx = pado.VertexCentricPLL(g, rank, bp_roots=16, batch=128)
    lab = orc.unw_label(g, rank, 16, 128)
    rng = np.random.Generator(np.random.PCG64(8))
    sizes = [1, 7, 300, 16384, 16385, 40000]
    pairs = [rng.integers(0, g.n, (2, k)).astype(np.uint32) for k in sizes]
    want = [orc.unw_query(lab, a, b) for a, b in pairs]
    wrong, stop = [], threading.Event()

    def ask(t):
        for i in range(60):
            j = (t + i) % len(sizes)
            if not np.array_equal(idx.query(*pairs[j]), want[j]):
                wrong.append((t, i, sizes[j]))

    def give_back():
        while not stop.is_set():
            _lib.check(_lib.lib.pado_set_scratch_cache(0))

    others = threading.Thread(target=give_back)
    threads = [threading.Thread(target=ask, args=(t,)) for t in range(12)]
    others.start()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    stop.set()
    others.join()
    assert not wrong
