"""Sorts where the device's SMs are not all to be had: on a stream of a green
context with a part of them, and where cooperative and cluster launches are
refused. No route may need more CTAs resident than the stream can hold."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import to_dev, to_np

pytestmark = pytest.mark.gpu

HOST_SORTS = """
import numpy as np, lsb_gb300 as lsb
r = np.random.default_rng(1)
for n in (9217, 20000, 100003, 700001, 1245184, 1300001):
    full = r.integers(0, 1 << 64, n, dtype=np.uint64)
    half = np.where(r.random(n) < 0.5, np.uint64(1 << 63) + (full & np.uint64(0xFFF)), full)  # runs to merge
    for keys in (full, half):
        a = np.empty((n, 2), np.uint64)
        a[:, 0], a[:, 1] = keys, np.arange(n)
        want = a[np.argsort(keys, kind="stable")]
        rc = lsb.load().lsb_sort_pairs_host(a.ctypes.data, n, 16, None)
        assert rc == 0, (n, lsb.status_string(rc))
        assert np.array_equal(a, want), n
print("sorted")
"""


def test_refused_launches(faked):
    """The one-launch sort and the run merges, each launch refused by the runtime."""
    assert "sorted" in faked(HOST_SORTS, FAKE_REFUSE="1")


class _Resource(ctypes.Structure):  # CUdevResource
    _fields_ = [("type", ctypes.c_int), ("pad", ctypes.c_ubyte * 92), ("sms", ctypes.c_uint), ("rest", ctypes.c_ubyte * 44)]


@pytest.fixture
def few_sms(cuda):
    """A stream on 16 SMs or a few more, and how many."""
    cuda.zeros(1, device="cuda")  # the device's context
    try:
        cu = ctypes.CDLL("libcuda.so.1")
        calls = [cu.cuDeviceGetDevResource, cu.cuDevSmResourceSplitByCount, cu.cuDevResourceGenerateDesc,
                 cu.cuGreenCtxCreate, cu.cuGreenCtxStreamCreate, cu.cuGreenCtxDestroy]
    except (OSError, AttributeError):
        pytest.skip("the driver has no green contexts")
    get, split, describe, create, stream_of, destroy = calls
    every, part, rest = _Resource(), _Resource(), _Resource()
    groups, desc, green, stream = ctypes.c_uint(1), ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    assert get(0, ctypes.byref(every), 1) == 0
    if split(ctypes.byref(part), ctypes.byref(groups), ctypes.byref(every), ctypes.byref(rest), 0, 16) != 0:
        pytest.skip("the device cannot be split")
    assert describe(ctypes.byref(desc), ctypes.byref(part), 1) == 0
    assert create(ctypes.byref(green), desc, 0, 1) == 0
    assert stream_of(ctypes.byref(stream), green, 1, 0) == 0
    yield cuda.cuda.ExternalStream(stream.value), part.sms
    cuda.cuda.synchronize()
    cu.cuStreamDestroy_v2(stream)
    destroy(green)


def test_stream_of_a_few_sms(lsb, cuda, oracle, few_sms):
    stream, sms = few_sms
    assert 16 <= sms < 100
    r = np.random.default_rng(2)
    for n in (5, 9217, 32768, 32769, 65537, 300007, 1245184, 1245185, 3000001):
        full = r.integers(0, 1 << 64, n, dtype=np.uint64)
        half = np.where(r.random(n) < 0.5, np.uint64(1 << 63) + (full & np.uint64(0xFFF)), full)
        for keys in (full, half, full & np.uint64(0xFF00FF)):
            a = np.stack([keys, np.arange(n, dtype=np.uint64)], axis=1)
            A = to_dev(a, cuda)
            B, ws = cuda.empty_like(A), lsb.alloc_workspace(n, 16)
            cuda.cuda.synchronize()
            lsb.sort_pairs(A, B, 16, workspace=ws, stream=stream)
            stream.synchronize()
            assert lsb.query(ws).device_status == 0
            assert np.array_equal(to_np(A), oracle.stable_sort_by_key(a)), n
    sizes = [5, 4608, 4609, 200003, 1000, 700001]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = int(off[-1])
    keys = np.where(r.random(n) < 0.5, np.uint64(77 << 50) + r.integers(0, 4096, n).astype(np.uint64),
                    r.integers(0, 1 << 64, n, dtype=np.uint64))
    a = np.stack([keys, np.arange(n, dtype=np.uint64)], axis=1)
    A, do = to_dev(a, cuda), cuda.from_numpy(off).cuda()
    B, ws = cuda.empty_like(A), lsb.alloc_segmented_workspace(n, len(sizes), 16)
    cuda.cuda.synchronize()
    lsb.sort_segmented(A, B, do, workspace=ws, stream=stream)
    stream.synchronize()
    assert lsb.query(ws).device_status == 0
    got = to_np(A)
    for s in range(len(sizes)):
        assert np.array_equal(got[off[s]:off[s + 1]], oracle.stable_sort_by_key(a[off[s]:off[s + 1]])), s
