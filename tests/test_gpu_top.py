"""The sort of whole arrays without going through every digit: arrays of one
shared-memory tile in one launch. Sizes at the edges of the tile shapes, key
sets that are even, clustered, duplicated, ordered and constant; bit-exact
against the oracle's stable sort, and the plan lsb_query reports."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import to_dev, to_np

pytestmark = pytest.mark.gpu


def _elems(keys):
    a = np.empty((len(keys), 2), dtype=np.uint64)
    a[:, 0] = keys
    a[:, 1] = np.arange(len(keys), dtype=np.uint64)
    return a


def key_sets(n, seed):
    """Named key arrays (uint64) of n elements: what a tile's bins meet."""
    r = np.random.default_rng(seed)
    full = r.integers(0, 1 << 64, n, dtype=np.uint64)
    yield "uniform", full
    yield "reverse", np.sort(full)[::-1].copy()
    yield "few", r.integers(0, 3, n).astype(np.uint64)
    yield "dups", full[r.integers(0, max(1, n // 30), n)]
    # an even spread and one cluster whose keys agree in all but their lowest bits
    c = full.copy()
    c[: n // 2] = np.uint64(1 << 60) + r.integers(0, 1000, n // 2).astype(np.uint64)
    yield "cluster", r.permutation(c)
    yield "extremes", np.where(r.random(n) < 0.5, np.uint64(0), np.uint64(2**64 - 1))
    yield "low_bits", (full & np.uint64(0xFFF)) | np.uint64(0xABCDEF << 40)
    # neighbours in the last bits of a wide range: the slots' key bits tie
    c = full[r.integers(0, max(1, n // 30), n)]
    yield "close_dups", c ^ r.integers(0, 2, n).astype(np.uint64)
    yield "close", np.repeat(full[: n // 2 + 1], 2)[:n] ^ r.integers(0, 2, n).astype(np.uint64)


def _run(lsb, cuda, a, bits):
    A = to_dev(a, cuda)
    B = cuda.empty_like(A)
    ws = lsb.alloc_workspace(a.shape[0], bits)
    lsb.sort_pairs(A, B, bits, workspace=ws)
    return to_np(A), lsb.query(ws)


@pytest.mark.parametrize("n", [2, 31, 33, 511, 513, 1000, 4607, 4608, 4609, 9215, 9216, 9217])
def test_one_tile(lsb, cuda, oracle, n):
    for name, keys in key_sets(n, n):
        a = _elems(keys)
        got, st = _run(lsb, cuda, a, 8)
        assert np.array_equal(got, oracle.stable_sort_by_key(a)), (n, name)
        diff = int(np.bitwise_or.reduce(keys ^ keys[0]))
        skipped = sum(1 << d for d in range(8) if not (diff >> (8 * d)) & 0xFF)
        runs = 8 - bin(skipped).count("1")
        assert (st.device_status, st.passes_planned, st.skipped_mask, st.passes_run, st.final_copy, st.n) == (
            0, 8, skipped, runs, runs & 1, n), (n, name)


def large_key_sets(n, seed):
    """Keys that leave short runs, long runs in order, long runs that must be merged, and none."""
    r = np.random.default_rng(seed)
    full = r.integers(0, 1 << 64, n, dtype=np.uint64)
    yield "uniform", full
    yield "sorted", np.sort(full)
    yield "reverse", np.sort(full)[::-1].copy()
    yield "equal", np.full(n, 0x0123456789ABCDEF, dtype=np.uint64)
    yield "low_20_bits", full & np.uint64(0xFFFFF)
    yield "offset_range", (full & np.uint64(0x3FFFFFFF)) + np.uint64(0x7FFFFFFFF0000000)
    # one key for half of the elements: its run is in order, or mixed with its neighbours
    yield "half_zero", np.where(r.random(n) < 0.5, np.uint64(0), full)
    h = np.where(r.random(n) < 0.5, np.uint64(1 << 63), full)
    h[r.integers(0, n, 50)] = np.uint64((1 << 63) + 1)
    yield "half_one_key_and_close_ones", h
    # three top halves: runs of a third of the array, all different below
    yield "three_prefixes", (r.integers(0, 3, n).astype(np.uint64) << np.uint64(61)) | (full >> np.uint64(32))
    # a narrow cluster that a sample sees little of, and keys far outside the others' block
    c = full.copy()
    k = max(n // 100, 20)
    c[r.permutation(n)[:k]] = np.uint64(0x5555000000000000) + r.integers(0, 1 << 30, k).astype(np.uint64)
    yield "cluster", c
    o = full & np.uint64(0xFFFFFFFF)
    o[r.integers(0, n, 3)] = np.uint64(2**64 - 1)
    o |= np.uint64(1 << 40)
    o[r.integers(0, n, 3)] = np.uint64(7)
    yield "outliers", o
    yield "equal_but_few", np.where(r.random(n) < 3e-4, full, np.uint64(0xFFFFFFFF00000000))
    yield "dups", full[r.integers(0, max(1, n // 3000), n)]


@pytest.mark.parametrize("n", [9217, 32768, 32769, 65537, 300007, 311296, 311297, 622593, 1245184, 1245185, (1 << 22) + 3])
def test_top_digits(lsb, cuda, oracle, n):
    """Runs of every kind, in one launch up to 8192 elements per SM (at the edges
    of its tile sizes on 152 SMs) and pass by pass above."""
    for name, keys in large_key_sets(n, n):
        a = _elems(keys)
        got, st = _run(lsb, cuda, a, 16)
        assert np.array_equal(got, oracle.stable_sort_by_key(a)), (n, name)
        diff = int(np.bitwise_or.reduce(keys ^ keys[0]))
        skipped = sum(1 << d for d in range(4) if not (diff >> (16 * d)) & 0xFFFF)
        assert (st.device_status, st.passes_planned, st.skipped_mask, st.n) == (0, 4, skipped, n), (n, name)


@pytest.mark.parametrize("variant", [0, 2])
def test_segments_of_every_kind(lsb, cuda, oracle, variant):
    """A batch whose arrays take each route: empty, one element, at the edges of
    the on-chip tile, one and two passes, and every kind of keys above."""
    parts = []
    for i, n in enumerate((0, 1, 2, 1000, 4607, 4608, 4609, 9217, 40000, 1100001)):
        sets = dict(large_key_sets(n, n)) if n > 9000 else dict(key_sets(n, n)) if n > 1 else {"one": np.arange(n, dtype=np.uint64)}
        for keys in sets.values() if n < 1000000 else [sets["uniform"], sets["dups"], sets["half_one_key_and_close_ones"]]:
            parts.append(_elems(keys))
    order = np.random.default_rng(variant).permutation(len(parts))
    parts = [parts[i] for i in order]
    off = np.zeros(len(parts) + 1, dtype=np.int64)
    off[1:] = np.cumsum([len(x) for x in parts])
    A = to_dev(np.concatenate(parts), cuda)
    B = cuda.empty_like(A)
    ws = lsb.alloc_segmented_workspace(A.shape[0], len(parts), 16)
    lsb.sort_segmented(A, B, cuda.from_numpy(off).cuda(), tuning=lsb.Tuning(digit_bits=16, variant=variant), workspace=ws)
    assert lsb.query(ws).device_status == 0
    got = to_np(A)
    for s, a in enumerate(parts):
        assert np.array_equal(got[off[s]:off[s + 1]], oracle.stable_sort_by_key(a)), (s, len(a))


@pytest.mark.parametrize("n,kind", [(280000001, "uniform"), (280000001, "cluster"), (1 << 28, "dense"), (566231040, "uniform")])
def test_runs_of_the_big_tile(lsb, cuda, n, kind):
    """Two passes where the usual tile would need three: runs of 4272 to 8640
    elements, and a run longer than any tile among them. Checked on the GPU: each
    value is the index of its key, and (key, value) rises strictly."""
    torch = cuda
    src = torch.randint(-2**63, 2**63 - 1, (n,), dtype=torch.int64, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    if kind == "cluster":
        src[::1000] = (src[::1000] & 0xFFFFFFFF) + (77 << 48)
    if kind == "dense":  # 28 bits of keys in a block of 29
        i = torch.arange(777777, 777777 + n, dtype=torch.int64, device="cuda")
        src = i ^ (i >> 3)
    A = torch.empty((n, 2), dtype=torch.int64, device="cuda")
    A[:, 0] = src
    A[:, 1] = torch.arange(n, dtype=torch.int64, device="cuda")
    B = torch.empty_like(A)
    ws = lsb.alloc_workspace(n, 16)
    lsb.sort_pairs(A, B, 16, workspace=ws)
    assert lsb.query(ws).device_status == 0
    del B
    for lo in range(0, n, 1 << 26):
        a = A[lo:min(n, lo + (1 << 26) + 1)]
        assert torch.equal(src[a[:, 1]], a[:, 0])
        k = a[:, 0] ^ (-2**63)
        assert bool(((k[1:] > k[:-1]) | ((k[1:] == k[:-1]) & (a[1:, 1] > a[:-1, 1]))).all())


@pytest.mark.parametrize("n", [1, 2, 8191, 8192, 8193, 70001])
@pytest.mark.parametrize("bits", [8, 16])
def test_one_digit(lsb, cuda, n, bits):
    """Single passes over the lowest, a constant and the highest digit, in one
    sub-pass or two, at the edges of the pass's tile; the source stays as it was."""
    r = np.random.default_rng(n)
    keys = r.integers(0, 1 << 64, n, dtype=np.uint64) & ~np.uint64(0xFFFF0000) | np.uint64(0x5A5A0000)
    a = _elems(keys)
    last = 64 // bits - 1
    for digit in (0, 16 // bits, last):
        src = to_dev(a, cuda)
        dst = cuda.empty_like(src)
        ws = cuda.empty(lsb.pass_workspace_bytes(n, bits), dtype=cuda.uint8, device="cuda")
        lsb.global_shuffle(src, dst, digit, bits, workspace=ws)
        d = (keys >> np.uint64(bits * digit)) & np.uint64((1 << bits) - 1)
        assert np.array_equal(to_np(dst), a[np.argsort(d, kind="stable")]), (n, bits, digit)
        assert np.array_equal(to_np(src), a)
        constant = int(len(np.unique(d)) == 1) if bits == 8 else 0
        st = lsb.query(ws)
        assert (st.device_status, st.skipped_mask, st.passes_run, st.n) == (0, constant, 1 - constant, n), (n, bits, digit)


@pytest.mark.parametrize("n", [8193, 16384 * 76 - 1, 16384 * 76, 3000001])
def test_histogram_of_16_bits(lsb, cuda, n):
    """Counters that go to the counts by atomics, and stored ones (from 2^14 keys
    per pair of CTAs, at the edge on 152 SMs); one digit is constant, one heavy."""
    r = np.random.default_rng(n)
    keys = r.integers(0, 1 << 64, n, dtype=np.uint64) & ~np.uint64(0xFFFF0000) | np.uint64(0x12340000)
    keys[r.random(n) < 0.5] &= np.uint64(0x0000FFFFFFFFFFFF)
    h = lsb.histogram(to_dev(_elems(keys), cuda), 16).cpu().numpy().reshape(4, 65536)
    for d in range(4):
        assert np.array_equal(h[d], np.bincount((keys >> np.uint64(16 * d)) & np.uint64(0xFFFF), minlength=65536)), (n, d)
