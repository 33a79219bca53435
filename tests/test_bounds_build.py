"""The bounds-checking build (PADO_DEBUG_BOUNDS) checks an access only where the
code makes it through UD_AT: the cover bitmaps and the padded rows of
bit-parallel distances are reached in no other way."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "parallel_distance_oracle_gb300" / "csrc"


def body(src: str, head: str) -> str:
    """The function whose definition starts with `head`, braces and all."""
    at = src.index(head)
    at = src.index("{", at)
    depth = 0
    for i in range(at, len(src)):
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        if depth == 0:
            return src[at:i + 1]
    raise AssertionError(head)


@pytest.mark.parametrize("head,accesses", [
    ("void bm_set(", 1), ("void bm_clear(", 1), ("bool bp_covered_lanes(", 2),
])
def test_helpers_use_checked_accesses(head, accesses):
    src = (CSRC / "unw_device.cuh").read_text()
    assert body(src, head).count("UD_AT(") == accesses


@pytest.mark.parametrize("name", ["unw_device.cuh", "unw.cu", "unw_many.cu"])
def test_no_pointer_arithmetic_beside_the_checks(name):
    """The arrays are only handed on (a batch parity's half is picked with bm_words)."""
    src = (CSRC / name).read_text()
    uses = re.findall(r"\b(?:d|bc|a)\.(?:bm|bpdp)\b\)?\s*[+\[][^;]*", src)
    assert all(re.match(r"d\.bm \+ \(+b(?: - 1\))? & 1\) \* bm_words\(", u) for u in uses), uses
