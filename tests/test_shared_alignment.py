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
