"""The work that programs give this library, as cases that can be timed: sorts
of one array from a thousand elements to 2^30, one distributed pass, batches of
uneven arrays, host arrays and the request loop, each through the Python
binding's public calls.

An array is an int64 CUDA tensor (n, 2): column 0 the key's bits (unsigned
order), column 1 the value. Values are the original indices, so stability
shows in the output.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "distributed-lsb_gb300"))

import lsb_gb300 as lsb  # noqa: E402

SIGN = -(1 << 63)
DISTS = ("uniform", "low32", "zipf", "equal", "nearly_sorted")


def listed():
    return [
        # the smallest sorts: a work queue's or a request's few thousand keys, where latency is all
        {"name": "sort_1k", "kind": "sort", "n": 1000, "bits": 16, "dist": "uniform"},
        {"name": "sort_64k", "kind": "sort", "n": 65537, "bits": 16, "dist": "uniform"},
        # ordinary sorts, at the digit widths the library offers for whole sorts
        {"name": "sort_1m_b8", "kind": "sort", "n": 1000003, "bits": 8, "dist": "uniform"},
        {"name": "sort_5m_b11", "kind": "sort", "n": 5000011, "bits": 11, "dist": "uniform"},
        # the benchmark's small configuration (2^24 uniform, the reference's 16-bit digits)
        {"name": "sort_16m", "kind": "sort", "n": 1 << 24, "bits": 16, "dist": "uniform"},
        # the benchmark's skew configuration: heavy duplicates, and an index-like key that is nearly sorted
        {"name": "sort_256m_zipf", "kind": "sort", "n": 1 << 28, "bits": 16, "dist": "zipf"},
        {"name": "sort_256m_nearly", "kind": "sort", "n": 1 << 28, "bits": 16, "dist": "nearly_sorted"},
        # the headline: 2^30 uniform
        {"name": "sort_1g", "kind": "sort", "n": 1 << 30, "bits": 16, "dist": "uniform"},
        # what a rank of the distributed sort does per pass on its block: the stable pass and the counts
        {"name": "rank_step_64m", "kind": "step", "n": (1 << 26) + 5, "bits": 16, "digit": 1, "dist": "uniform"},
        # many independent arrays of uneven sizes as one captured batch (the benchmark's size law)
        {"name": "batch_512", "kind": "batch", "nseg": 512, "lo": 10.0, "hi": 22.0, "mix": 1, "dist": "uniform"},
        # an array in (page-locked) host memory, sorted through the one-call host entry point
        {"name": "host_1m5", "kind": "host", "n": 1500007, "bits": 16, "dist": "uniform"},
        # the request loop: requests of mixed sizes from host buffers, admitted as they come
        {"name": "serve_24", "kind": "serve", "requests": 24, "lo": 10.0, "hi": 20.0, "mix": 2, "bits": 16},
    ]


def _log_size(rng, lo, hi):
    """An integer from 2^lo to 2^hi, spread over the logarithm; most are odd."""
    n = int(2.0 ** rng.uniform(lo, hi))
    return n | 1 if rng.random() < 0.75 else n


def draw(rng):
    kind = rng.choice(("sort", "sort", "sort", "sort", "step", "batch", "host", "serve"))
    if kind == "sort":
        dist = rng.choice(("uniform", "uniform", "uniform", "zipf", "low32", "nearly_sorted", "equal"))
        # 11-bit digits stay below 2^28: above, such a sort costs more than the largest listed one
        bits = rng.choice((16, 16, 8, 11))
        return {"kind": "sort", "n": _log_size(rng, 10.0, 28.0 if bits == 11 else 29.0), "bits": bits, "dist": dist}
    if kind == "step":
        bits = rng.choice((16, 8))
        return {"kind": "step", "n": _log_size(rng, 16.0, 26.0), "bits": bits,
                "digit": rng.randrange(64 // bits), "dist": rng.choice(("uniform", "uniform", "zipf"))}
    if kind == "batch":
        return {"kind": "batch", "nseg": int(2.0 ** rng.uniform(3.0, 9.0)), "lo": 10.0, "hi": round(rng.uniform(14.0, 22.0), 2),
                "mix": rng.randrange(1 << 20), "dist": rng.choice(("uniform", "uniform", "zipf"))}
    if kind == "host":
        return {"kind": "host", "n": _log_size(rng, 10.0, 22.0), "bits": rng.choice((16, 8)),
                "dist": rng.choice(("uniform", "zipf", "nearly_sorted"))}
    return {"kind": "serve", "requests": rng.randrange(4, 33), "lo": 10.0, "hi": round(rng.uniform(14.0, 20.0), 2),
            "mix": rng.randrange(1 << 20), "bits": 16}


def _sizes(count, lo, hi, mix):
    """floor(2^U(lo, hi)) for each of `count` arrays: the size law of the batch and serving benchmarks."""
    return np.floor(2.0 ** np.random.default_rng(mix).uniform(lo, hi, count)).astype(np.int64)


def _keys(n, dist, seed):
    """n keys of one of the benchmark's five distributions, on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))

    def uniform(m):
        return torch.randint(SIGN, (1 << 63) - 1, (m,), dtype=torch.int64, device="cuda", generator=g)

    if dist == "uniform":
        return uniform(n)
    if dist == "low32":
        return uniform(n) & 0xFFFFFFFF
    if dist == "equal":
        return uniform(1).expand(n).contiguous()
    if dist == "nearly_sorted":
        # i ^ (i >> 3) around a start of the seed's own: the keys of a log that is nearly in order
        start = int(torch.randint(0, 1 << 20, (1,), device="cuda", generator=g).item())
        i = torch.arange(start, start + n, dtype=torch.int64, device="cuda")
        return i ^ (i >> 3)
    # Zipf(1.1) ranks over 2^20 distinct keys
    distinct = uniform(1 << 20)
    cdf = torch.cumsum(torch.arange(1, (1 << 20) + 1, dtype=torch.float64, device="cuda") ** -1.1, 0)
    cdf /= cdf[-1].clone()
    out = torch.empty(n, dtype=torch.int64, device="cuda")
    for lo in range(0, n, 1 << 26):
        hi = min(n, lo + (1 << 26))
        u = torch.rand(hi - lo, dtype=torch.float64, device="cuda", generator=g)
        out[lo:hi] = distinct[torch.searchsorted(cdf, u).clamp_(max=(1 << 20) - 1)]
    return out


def _array(n, dist, seed):
    a = torch.empty((n, 2), dtype=torch.int64, device="cuda")
    a[:, 0] = _keys(n, dist, seed)
    a[:, 1] = torch.arange(n, dtype=torch.int64, device="cuda")
    return a


class _Serving:
    """A program around the request loop: its server, its requests and their page-locked buffers."""

    def __init__(self, case, seed):
        sizes = _sizes(case["requests"], case["lo"], case["hi"], case["mix"])
        self.fresh = [_array(int(s), "uniform", seed * 1000 + i).cpu() for i, s in enumerate(sizes)]
        self.buffers = [torch.empty_like(f).pin_memory() for f in self.fresh]
        self.server = lsb.Server(slots=4, digit_bits=case["bits"], hbm_budget_bytes=8 << 30)

    def __del__(self):
        if hasattr(self, "server"):
            self.server.close()


def prepare(case, seed):
    """Inputs from the seed, and what a program keeps between calls: scratch array, workspace, tuned plan, graph, server."""
    kind = case["kind"]
    if kind == "serve":
        return {"case": case, "serving": _Serving(case, seed)}
    if kind == "host":
        fresh = _array(case["n"], case["dist"], seed).cpu()
        return {"case": case, "fresh": fresh, "buffer": torch.empty_like(fresh).pin_memory()}
    if kind == "batch":
        sizes = _sizes(case["nseg"], case["lo"], case["hi"], case["mix"])
        off = np.zeros(len(sizes) + 1, dtype=np.int64)
        off[1:] = np.cumsum(sizes)
        n = int(off[-1])
        fresh = _array(n, case["dist"], seed)
        a, b = torch.empty_like(fresh), torch.empty_like(fresh)
        tuning = lsb.tune_segmented(off)
        ws = lsb.alloc_segmented_workspace(n, len(sizes), tuning.digit_bits)
        offsets = torch.from_numpy(off).cuda()
        torch.cuda.synchronize()
        return {"case": case, "fresh": fresh, "a": a, "graph": lsb.SegmentedGraph(a, b, offsets, tuning, ws)}
    n, bits = case["n"], case["bits"]
    fresh = _array(n, case["dist"], seed)
    if kind == "step":
        ws = torch.empty(lsb.pass_workspace_bytes(n, bits), dtype=torch.uint8, device="cuda")
        return {"case": case, "fresh": fresh, "a": torch.empty_like(fresh), "ws": ws}
    return {"case": case, "fresh": fresh, "a": torch.empty_like(fresh), "b": torch.empty_like(fresh),
            "ws": lsb.alloc_workspace(n, bits)}


def run(state):
    """One pass. The sorts work in place, so the new data is first put into the array, as a program that receives it does."""
    case = state["case"]
    kind = case["kind"]
    if kind == "sort":
        state["a"].copy_(state["fresh"])
        lsb.sort_pairs(state["a"], state["b"], case["bits"], workspace=state["ws"])
        return state["a"]
    if kind == "step":
        lsb.global_shuffle(state["fresh"], state["a"], case["digit"], case["bits"], workspace=state["ws"])
        return state["a"], lsb.histogram(state["fresh"], case["bits"])
    if kind == "batch":
        state["a"].copy_(state["fresh"])
        state["graph"].launch()
        return state["a"]
    if kind == "host":
        state["buffer"].copy_(state["fresh"])
        lsb.sort_pairs_host(state["buffer"], case["bits"])
        return state["buffer"]
    s = state["serving"]
    ids = []
    for f, h in zip(s.fresh, s.buffers):
        h.copy_(f)
        ids.append(s.server.submit_host(h))
    for i in ids:
        s.server.wait(i)
    return list(s.buffers)


def work(case):
    """Each element is read once and written once, 16 bytes each way; a pass's counts are written once."""
    kind = case["kind"]
    if kind == "batch":
        n = int(_sizes(case["nseg"], case["lo"], case["hi"], case["mix"]).sum())
    elif kind == "serve":
        n = int(_sizes(case["requests"], case["lo"], case["hi"], case["mix"]).sum())
    else:
        n = case["n"]
    counts = 0
    if kind == "step":
        counts = math.ceil(64 / case["bits"]) * (1 << case["bits"]) * 8
    return {"bytes": 32 * n + counts, "flops": 0}


def _sorted(a, key):
    """Rows of `a` in the stable order of `key`'s 64 bits, taken as unsigned."""
    return a[torch.sort(key ^ SIGN, stable=True)[1]]


def exact(case, seed):
    """The same outputs from torch's stable sort."""
    kind = case["kind"]
    if kind == "serve":
        sizes = _sizes(case["requests"], case["lo"], case["hi"], case["mix"])
        arrays = [_array(int(s), "uniform", seed * 1000 + i) for i, s in enumerate(sizes)]
        return [_sorted(a, a[:, 0]).cpu() for a in arrays]
    if kind == "batch":
        sizes = _sizes(case["nseg"], case["lo"], case["hi"], case["mix"])
        a = _array(int(sizes.sum()), case["dist"], seed)
        return torch.cat([_sorted(part, part[:, 0]) for part in torch.split(a, [int(s) for s in sizes])])
    if case["n"] > 1 << 28:
        return None
    a = _array(case["n"], case["dist"], seed)
    if kind == "step":
        bits, mask = case["bits"], (1 << case["bits"]) - 1
        digits = [(a[:, 0] >> (bits * d)) & mask for d in range(64 // bits)]
        counts = torch.stack([torch.bincount(d, minlength=1 << bits) for d in digits])
        return _sorted(a, digits[case["digit"]]), counts
    out = _sorted(a, a[:, 0])
    return out.cpu() if kind == "host" else out
