"""Shared memory that is accessed in 16-byte pieces is declared with that alignment (no
GPU: the declarations are read from the sources; where the compiler happens to put an
array says nothing about the next build)."""
from __future__ import annotations

import re

from conftest import PKG_NAME, ROOT

CSRC = ROOT / PKG_NAME / "csrc"


def test_ordered_sums_read_aligned_pairs():
    src = (CSRC / "tke.cu").read_text()
    assert "reinterpret_cast<const double2 *>(v)" in src  # the pairs that ordered_sums reads
    assert re.search(r"struct alignas\(16\) SumSmem\b", src)


def test_bulk_copies_land_in_aligned_rows():
    arrays = 0
    for src in sorted(CSRC.glob("pair_*.cu")):  # the kernels whose rows bulk copies bring in
        for decl in re.findall(r"extern __shared__ ([^;]*);", src.read_text()):
            assert "__align__(16)" in decl, (src.name, decl)
            arrays += 1
    assert arrays == 2  # one a precision
