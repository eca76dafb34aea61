"""The pass kernels by single passes: whole sorts take kernels of their own unless one
is asked for by name, so what they did for the kernels of 9 to 11 bits (and of the
widths below 8) is done here through lsb_pass, and through a sort that is chained
from it."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import to_dev, to_np

pytestmark = pytest.mark.gpu

TILE = 8192
DISTS = [0, 1, 2, 3, 4]


@pytest.mark.parametrize("variant", ["0", "4"])
@pytest.mark.parametrize("bits", [9, 10, 11])
def test_wide_bins_at_tile_edges(lsb, cuda, oracle, monkeypatch, bits, variant):
    monkeypatch.setenv("LSB_ONESWEEP_VARIANT", variant)
    for n in (1, 2, 31, TILE - 1, TILE, TILE + 1, 3 * TILE + 17, 40 * TILE + 5):
        for dist in DISTS:
            a = oracle.generate(n, dist, n % 13)
            src = to_dev(a, cuda)
            cur, other = src.clone(), cuda.empty_like(src)
            for d in range(lsb.num_passes(bits)):  # the whole sort, a pass at a time
                lsb.global_shuffle(cur, other, d, bits)
                cur, other = other, cur
                if d in (0, lsb.num_passes(bits) - 1):
                    dst = cuda.empty_like(src)
                    lsb.global_shuffle(src, dst, d, bits)
                    assert np.array_equal(to_np(dst), oracle.global_shuffle(a, d, bits)), (bits, n, dist, d)
            assert np.array_equal(to_np(cur), oracle.stable_sort_by_key(a)), (bits, n, dist)


@pytest.mark.parametrize("bits", [1, 4, 5, 8, 12, 13, 15, 16])
def test_other_widths_chained(lsb, cuda, oracle, bits):
    for dist, n in ((0, 70001), (2, TILE + 1), (4, 3 * TILE)):
        a = oracle.generate(n, dist, 3)
        cur = to_dev(a, cuda)
        other = cuda.empty_like(cur)
        for d in range(lsb.num_passes(bits)):
            lsb.global_shuffle(cur, other, d, bits)
            cur, other = other, cur
        assert np.array_equal(to_np(cur), oracle.stable_sort_by_key(a)), (bits, dist)
