"""bench.py's roofline of a whole sort: the bytes a sort cannot do without."""
from __future__ import annotations

import sys

import pytest

from conftest import ROOT


def test_sort_roofline_counts_each_element_once_in_and_once_out():
    sys.path.insert(0, ROOT)
    import bench

    r = bench.sort_roofline(1 << 30, 30.84, 6779.0)  # no fraction above one, whatever the digit width
    assert r["algorithmic_bytes_per_element"] == 32
    assert r["achieved_gbs"] == pytest.approx(32 * (1 << 30) / 30.84e-3 / 1e9, abs=0.1)
    assert r["frac"] == pytest.approx(r["achieved_gbs"] / 6779.0, abs=1e-3) and r["frac"] < 1
