"""The profile of a build puts the bytes that a kernel counts into the row of its
launches (the labeling loops' phases excepted, which have rows of their own)."""
import ctypes as C

import pytest

from parallel_distance_oracle_gb300 import graphs as G

pytestmark = pytest.mark.gpu

PHASES = {"pull_kernel", "mark_kernel", "w_pull_kernel", "w_mark_kernel"}


def test_counted_bytes_are_in_launched_rows(cuda_ok):
    from parallel_distance_oracle_gb300 import _lib, pado
    g = G.rmat(11, 8, 5)
    _lib.lib.pado_profile_read(None, 0, 1)  # clears what earlier calls left in the table
    _lib.check(_lib.lib.pado_profile(1))
    try:
        idx = pado.VertexCentricPLL(g, G.degree_rank(g), bp_roots=16, batch=64)
        idx.query([1, 2], [3, 4])
        buf = C.create_string_buffer(1 << 16)
        _lib.lib.pado_profile_read(buf, len(buf), 1)
    finally:
        _lib.check(_lib.lib.pado_profile(0))
    rows = {ln.split()[0]: (int(ln.split()[1]), int(ln.split()[3])) for ln in buf.value.decode().splitlines()}
    counted = {k for k, (_, nbytes) in rows.items() if nbytes and "." not in k}
    assert {"bp_loop_kernel", "query_unw_kernel"} <= counted
    assert all(rows[k][0] for k in counted - PHASES), rows
