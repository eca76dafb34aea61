"""A workspace sized for the largest array serves every smaller one."""
from __future__ import annotations

import json

import numpy as np
import pytest

from conftest import to_dev, to_np

SIZES = """
import json, lsb_gb300 as lsb
sms, bits = {sms}, {bits}
edges = [m * sms for m in (1024, 2048, 4096, 8192)] + [9216, 32768]
sizes = sorted({{n + d for n in edges for d in (-1, 0, 1, 2047, 2049)}} | {{1, 2, 1000, 400000, 520000, 600000, 2000003, 1 << 24}})
print(json.dumps([[n, lsb.workspace_bytes(n, bits)] for n in sizes if n > 0]))
"""


@pytest.mark.parametrize("sms", [152, 148, 20])
@pytest.mark.parametrize("bits", [4, 8, 12, 16])
def test_need_never_falls_with_the_size(faked, sms, bits):
    """At each step of the tile sizes of the one-launch sort (2048, 4096 and 8192
    elements for every SM) on a faked device."""
    rows = json.loads(faked(SIZES.format(sms=sms, bits=bits), FAKE_SMS=str(sms)))
    for (n0, w0), (n1, w1) in zip(rows, rows[1:]):
        assert w1 >= w0, (n0, w0, n1, w1)


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [4, 8, 12])
def test_one_workspace_for_all_sizes(lsb, cuda, oracle, bits):
    for largest in (311297, 400000, 520000, 622593):
        ws = lsb.alloc_workspace(largest, bits)
        for n in (largest, 311296, 300007, 40000, 9217, 5):
            a = oracle.generate(n, oracle.DIST_UNIFORM, n)
            A = to_dev(a, cuda)
            lsb.sort_pairs(A, cuda.empty_like(A), bits, workspace=ws)
            assert lsb.query(ws).device_status == 0
            assert np.array_equal(to_np(A), oracle.stable_sort_by_key(a)), (largest, n)
