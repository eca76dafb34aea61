"""Keys as programs have them: signs, sentinels, tags, pairs, text, exponents,
clusters, bits that never vary. Every route of a whole sort and of a batch meets
them (one CTA, one cluster, one launch with each tile size, pass by pass with one
to eight digits, each last step), checked element by element; and their runs are not
left to the merges."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIGN = -(1 << 63)


def _families(torch, n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def ints(lo, hi, m=n):
        return torch.randint(lo, hi, (m,), dtype=torch.int64, device="cuda", generator=g)

    def unit():
        return torch.rand(n, dtype=torch.float64, device="cuda", generator=g)

    u = ints(SIGN, (1 << 63) - 1)
    yield "sign_8", ints(-128, 128)
    yield "sign_24", ints(-(1 << 24), 1 << 24)
    yield "sign_32_flipped", ints(-(1 << 31), 1 << 31) ^ SIGN
    yield "sign_40", ints(-(1 << 40), 1 << 40)
    yield "tag_32", (ints(0, 4) << 62) | ints(0, 1 << 32)
    yield "tag_16", (ints(0, 3) << 60) | ints(0, 1 << 16)
    yield "sentinels", torch.where(unit() < 0.01, -1, ints(0, 1 << 32))
    yield "few_sentinels", torch.where(unit() < 2e-4, -1, ints(0, 1 << 32))
    yield "pairs", (ints(0, 1 << 10) << 32) | ints(0, 1 << 24)
    yield "two_clusters", torch.where(unit() < 0.5, 1 << 20, 1 << 60) + ints(0, 1 << 20)
    yield "clusters", ints(SIGN, (1 << 63) - 1, 100)[ints(0, 100)] + ints(0, 1 << 16)
    yield "half_cluster", torch.where(unit() < 0.5, u, (5 << 58) + ints(0, 1 << 20))
    yield "exponents", torch.pow(2.0, unit() * 62.9).long()
    yield "normal", torch.randn(n, dtype=torch.float64, device="cuda", generator=g).view(torch.int64)
    yield "text", sum(ints(97, 123) << (8 * k) for k in range(8))
    yield "nibbles", u & 0x0F0F0F0F0F0F0F0F
    yield "scattered_bits", u & 0x1111111111111111
    yield "alternate_bytes", u & 0x00FF00FF00FF00FF
    yield "duplicates", u[ints(0, max(1, n // 30))]


def _array(torch, keys):
    a = torch.empty((keys.shape[0], 2), dtype=torch.int64, device="cuda")
    a[:, 0] = keys
    a[:, 1] = torch.arange(keys.shape[0], dtype=torch.int64, device="cuda")
    return a


@pytest.mark.parametrize("n", [3001, 9216, 9217, 20001, 32769, 200003, 311297, 622593, 1100001, 1245184, 1245185, 2000003,
                               (1 << 22) + 1, 17000001])
def test_sorted_stably(lsb, cuda, n):
    torch = cuda
    B = torch.empty((n, 2), dtype=torch.int64, device="cuda")
    ws = lsb.alloc_workspace(n, 8)
    for name, keys in _families(torch, n, n):
        a = _array(torch, keys)
        A = a.clone()
        lsb.sort_pairs(A, B, 8, workspace=ws)
        st = lsb.query(ws)
        assert (st.device_status, st.n) == (0, n), name
        assert lsb.verify(a, A) == 0, name
        k = keys ^ keys[0]
        runs = sum(bool(((k >> (8 * d)) & 255).any()) for d in range(8))
        assert st.passes_run == runs, name


@pytest.mark.parametrize("variant", [0, 2])
def test_batches_sorted_stably(lsb, cuda, variant):
    """Arrays of every family in one batch: 1000 elements to 300000, each size with each kind."""
    torch = cuda
    parts = []
    for n in (1000, 4609, 20001, 300001):
        parts += [keys for _, keys in _families(torch, n, n + variant)]
    off = np.concatenate([[0], np.cumsum([len(p) for p in parts])]).astype(np.int64)
    a = _array(torch, torch.cat(parts))
    A, B, do = a.clone(), torch.empty_like(a), torch.from_numpy(off).cuda()
    ws = lsb.alloc_segmented_workspace(a.shape[0], len(parts), 8)
    lsb.sort_segmented(A, B, do, tuning=lsb.Tuning(digit_bits=8, variant=variant), workspace=ws)
    assert lsb.query(ws).device_status == 0
    for s, keys in enumerate(parts):
        got = A[off[s]:off[s + 1]]
        order = torch.sort(keys ^ SIGN, stable=True)[1]
        assert torch.equal(got[:, 0], keys[order]) and torch.equal(got[:, 1] - int(off[s]), order), s


@pytest.mark.parametrize("far", [False, True, "five", "clamped"])
def test_many_digits_of_a_large_array(lsb, cuda, far):
    """Above 2^26 elements (a larger sample): half of the keys even, half in a cluster
    of 2^20 neighbours, so that every digit is passed over; a block with a gap in it
    and keys far outside; a cluster of 2^32, which five or six digits part, in the
    whole range and in a block with keys outside, which are clamped to it. Also as one
    array of a batch."""
    torch = cuda
    n = (1 << 26) + 12345
    g = torch.Generator(device="cuda")
    g.manual_seed(n + len(str(far)))
    u = torch.randint(SIGN, (1 << 63) - 1, (n,), dtype=torch.int64, device="cuda", generator=g)
    even = torch.rand(n, device="cuda", generator=g) < 0.5
    near = (5 << 40) + (u & 0xFFFFF)
    if far in ("five", "clamped"):
        keys = torch.where(even, u if far == "five" else u & 0xFFFFFFFFFFFFFF, (5 << 40) + (u & 0xFFFFFFFF))
        if far == "clamped":
            keys[[5, n // 2, n - 7]] = torch.tensor([-1, -2, 1 << 62], dtype=torch.int64, device="cuda")
    elif far:  # a block of 47 bits that three keys are outside of
        keys = torch.where(even, (u & 0x7F) << 40, near & 0x7FFFFFFFFFF)
        keys[[5, n // 2, n - 7]] = torch.tensor([-1, -2, 1 << 62], dtype=torch.int64, device="cuda")
    else:
        keys = torch.where(even, u, near)
    a = _array(torch, keys)
    A, B = a.clone(), torch.empty_like(a)
    ws = lsb.alloc_workspace(n, 16)
    lsb.sort_pairs(A, B, 16, workspace=ws)
    assert lsb.query(ws).device_status == 0 and lsb.verify(a, A) == 0
    del ws
    off = torch.tensor([0, n - 100003, n], dtype=torch.int64, device="cuda")
    ws = lsb.alloc_segmented_workspace(n, 2, 16)
    A.copy_(a)
    lsb.sort_segmented(A, B, off, workspace=ws)
    assert lsb.query(ws).device_status == 0
    for lo, hi in ((0, n - 100003), (n - 100003, n)):
        got = A[lo:hi]
        assert torch.equal(keys[got[:, 1]], got[:, 0]) and int(got[:, 1].min()) == lo and int(got[:, 1].max()) == hi - 1
        k = got[:, 0] ^ SIGN
        assert bool(((k[1:] > k[:-1]) | ((k[1:] == k[:-1]) & (got[1:, 1] > got[:-1, 1]))).all())


@pytest.mark.parametrize("n", [(1 << 22) + 1, (1 << 24) + 1])
def test_passes_not_merges(lsb, cuda, n):
    """The digits are chosen so that runs fit on chip: what is left to the merges of
    longer runs (a hundredth of the keys at most) takes less than a fifth of the time."""
    torch = cuda
    A, B = (torch.empty((n, 2), dtype=torch.int64, device="cuda") for _ in range(2))
    ws = lsb.alloc_workspace(n, 8)
    for name, keys in _families(torch, n, 3):
        a = _array(torch, keys)
        for timed in (False, True):
            A.copy_(a)
            torch.cuda.synchronize()
            lsb.profile_enable(timed)
            lsb.sort_pairs(A, B, 8, workspace=ws)
            torch.cuda.synchronize()
        lsb.profile_enable(False)
        ms = {k: v[1] for k, v in lsb.profile_read().items()}
        assert ms["top_merge"] < 0.2 * sum(ms.values()), (name, ms)


@pytest.mark.parametrize("kind", ["thousandfold", "clusters"])
def test_big_tile_only_where_it_fits(lsb, cuda, kind):
    """1.5 million keys of a thousand equals each, or in a hundred clusters: one pass
    leaves many of their runs longer than any tile, so that the sample has to say no
    to the tile that takes the runs of even keys after one pass."""
    torch = cuda
    n = 1500001
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    few = torch.randint(SIGN, (1 << 63) - 1, (n // 1000 if kind == "thousandfold" else 100,), dtype=torch.int64, device="cuda", generator=g)
    keys = few[torch.randint(0, few.shape[0], (n,), device="cuda", generator=g)]
    if kind == "clusters":
        keys = keys + torch.randint(0, 1 << 32, (n,), dtype=torch.int64, device="cuda", generator=g)
    a = _array(torch, keys)
    A, B = a.clone(), torch.empty_like(a)
    ws = lsb.alloc_workspace(n, 16)
    for timed in (False, True):
        A.copy_(a)
        torch.cuda.synchronize()
        lsb.profile_enable(timed)
        lsb.sort_pairs(A, B, 16, workspace=ws)
        torch.cuda.synchronize()
    lsb.profile_enable(False)
    ms = {k: v[1] for k, v in lsb.profile_read().items()}
    assert lsb.query(ws).device_status == 0 and lsb.verify(a, A) == 0
    assert ms["top_merge"] < 0.2 * sum(ms.values()), ms


@pytest.mark.parametrize("n,passes", [(1500001, 1), (2000003, 2), ((1 << 27) + 1, 2)])
def test_profile_counts_passes(lsb, cuda, n, passes):
    """Launches that find nothing to do are not among the pass launches whose mean
    time a profile gives: even keys make all of those."""
    torch = cuda
    a = _array(torch, torch.randint(SIGN, (1 << 63) - 1, (n,), dtype=torch.int64, device="cuda"))
    A, B = a.clone(), torch.empty_like(a)
    lsb.profile_enable(True)
    lsb.sort_pairs(A, B, 16)
    torch.cuda.synchronize()
    lsb.profile_enable(False)
    assert lsb.profile_read()["onesweep_scatter"][0] == passes
    assert lsb.verify(a, A) == 0


@pytest.mark.parametrize("n", [1, 8193, 8192 * 152 + 77, 3000001])
def test_pass_over_a_constant_digit(lsb, cuda, n):
    """A single pass whose digit is the same in all keys copies the array, over more
    than one round of every CTA too; the source stays as it was."""
    torch = cuda
    a = _array(torch, torch.randint(0, 1 << 32, (n,), dtype=torch.int64, device="cuda"))
    src, dst = a.clone(), torch.zeros_like(a)
    ws = torch.empty(lsb.pass_workspace_bytes(n, 8), dtype=torch.uint8, device="cuda")
    lsb.global_shuffle(src, dst, 5, 8, workspace=ws)
    st = lsb.query(ws)
    assert (st.device_status, st.skipped_mask, st.passes_run) == (0, 1, 0)
    assert torch.equal(dst, a) and torch.equal(src, a)
