"""Algorithmic bytes that bench.py charges an ingest's scatter launches: 16 a key
and pass, 12 in the last, over as many 8-bit passes as two ids need."""
import pytest

import bench


@pytest.mark.parametrize("n,passes", [(1, 1), (2, 1), (16, 1), (17, 2), (1 << 13, 4), (1 << 16, 4), ((1 << 16) + 1, 5),
                                      (1_048_106, 5), (1 << 20, 5), ((1 << 20) + 1, 6), (1 << 24, 6)])
def test_scatter_bytes(n, passes):
    m = 10_000_000
    got = bench.ingest_kernel_bytes("rs_scatter_kernel", m, n)
    assert abs(got * passes - ((passes - 1) * 16 + 12) * 2 * m) < passes
