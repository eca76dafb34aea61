"""What the library keeps for a device (kernel attributes among it) is good for
every context: sorts in a second context of the same device, in the first one after
that, and after cudaDeviceReset."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu

SORTS = """
import ctypes, numpy as np, lsb_gb300 as lsb
L = lsb.load()
cu = ctypes.CDLL("libcuda.so.1")
def ok(rc): assert rc == 0, rc
ctx, dev = ctypes.c_void_p(), ctypes.c_int()

def sorts():
    r = np.random.default_rng(3)
    for n in (1000, 5000, 20000, 100000, 1500001):
        a = np.empty((n, 2), np.uint64)
        a[:, 0], a[:, 1] = r.integers(0, 1 << 64, n, dtype=np.uint64), np.arange(n)
        need = lsb.workspace_bytes(n, 16)
        bufs = []
        for size in (16 * n, 16 * n, need):
            p = ctypes.c_uint64()
            ok(cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(size)))
            bufs.append(p)
        A, B, ws = (p.value for p in bufs)
        ok(cu.cuMemcpyHtoD_v2(bufs[0], a.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(16 * n)))
        rc = L.lsb_sort_pairs(A, B, n, 16, ws, need, None)
        assert rc == 0, (n, lsb.status_string(rc))
        ok(cu.cuCtxSynchronize())
        got = np.empty_like(a)
        ok(cu.cuMemcpyDtoH_v2(got.ctypes.data_as(ctypes.c_void_p), bufs[0], ctypes.c_size_t(16 * n)))
        assert np.array_equal(got, a[np.argsort(a[:, 0], kind="stable")]), n
        for p in bufs:
            ok(cu.cuMemFree_v2(p))

ok(cu.cuInit(0))
ok(cu.cuDevicePrimaryCtxRetain(ctypes.byref(ctx), 0))
ok(cu.cuCtxSetCurrent(ctx))
sorts()
for i in range(2):
    other = ctypes.c_void_p()
    ok(cu.cuCtxCreate_v2(ctypes.byref(other), 0, 0))
    sorts()
    if i:  # the first one again while the second is there
        ok(cu.cuCtxSetCurrent(ctx))
        sorts()
        ok(cu.cuCtxSetCurrent(other))
    ok(cu.cuCtxDestroy_v2(other))
ok(cu.cuCtxSetCurrent(ctx))
sorts()
rt = ctypes.CDLL("libcudart.so.13")  # the library's
for _ in range(2):
    ok(rt.cudaDeviceReset())
    ok(rt.cudaFree(None))
    sorts()
print("sorted")
"""


def test_second_context(lsb, cuda):
    r = subprocess.run([sys.executable, "-c", SORTS], capture_output=True, text=True, timeout=300, cwd=ROOT,
                       env={**os.environ, "PYTHONPATH": PKG + os.pathsep + ROOT})
    assert r.returncode == 0 and "sorted" in r.stdout, r.stdout + r.stderr
