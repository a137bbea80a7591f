"""Short key-value arrays in one launch (short_pairs.cuh) at their edges: the
smallest and largest sizes of each number of regions, pointers off the 16- and
32-byte boundaries, equal keys in a region (the bitonic sort of its words),
identifiers just past a power of two, regions that overflow and keys outside
the sampled bits (the digit passes then run); keys and values equal to the
oracle's stable sort (sorts are exact: no tolerance)."""

import numpy as np
import pytest

from _oracle import KEY_BYTES, raw_keys
from gpu_util import gpu_sort

pytestmark = pytest.mark.gpu


def _eq(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


def _check(gb, cuda, oracle, kt, raw, vb, desc, **kw):
    vals = np.arange(raw.shape[0], dtype=np.uint32 if vb == 4 else np.uint64)[::-1].copy()
    k, v = gpu_sort(gb, cuda, kt, raw, desc, vals, garbage_workspace=True, **kw)
    ek, ev = oracle.sort(kt, raw, desc, vals)
    assert _eq(k, ek)
    assert _eq(v, ev)


@pytest.mark.parametrize("kt", ["u32", "i32", "u64", "i64"])
@pytest.mark.parametrize("n", [2047, 2048, 2049, 4097, 65536, 270001, 275001, 500001, 655001, 660001, 1130001,
                               1180001, 2280001, 2400001])
def test_sizes(gb, cuda, oracle, kt, n):
    if KEY_BYTES[kt] == 8 and n > 1_200_000:
        n //= 2
    _check(gb, cuda, oracle, kt, raw_keys(kt, n, seed=n), 4 if n & 1 else 8, bool(n & 2))


@pytest.mark.parametrize("kt", ["u32", "u64"])
@pytest.mark.parametrize("how", ["few", "pairs_of_equals", "all_equal", "ids", "past_a_power", "outlier", "two_heaps",
                                 "sorted", "low_bits"])
@pytest.mark.parametrize("n", [5003, 262147])
def test_spreads(gb, cuda, oracle, kt, how, n):
    raw = raw_keys(kt, n, seed=n)
    rng = np.random.default_rng(n)
    t = raw.dtype.type
    if how == "few":  # a thousand distinct keys: crowded sub-buckets
        raw = raw[:1000][rng.integers(0, 1000, n)]
    elif how == "pairs_of_equals":
        raw = raw[: n // 40][rng.integers(0, n // 40, n)]
    elif how == "all_equal":
        raw[:] = raw[0]
    elif how == "ids":
        raw = rng.integers(0, n, n).astype(raw.dtype)
    elif how == "past_a_power":  # one key has a bit that the sample misses
        raw = rng.integers(0, 1 << 12, n).astype(raw.dtype)
        raw[n // 2 + 1] = t(1 << 12)
    elif how == "outlier":
        raw = rng.integers(0, 1 << 16, n).astype(raw.dtype)
        raw[n // 2 + 1] = t((1 << (8 * KEY_BYTES[kt] - 1)) + 5)
    elif how == "two_heaps":
        raw = (raw >> t(8 * KEY_BYTES[kt] - 10)) | (t(1) << t(8 * KEY_BYTES[kt] - 1)) * (raw & t(1))
    elif how == "sorted":
        raw = np.sort(raw)
    elif how == "low_bits":
        raw = raw & t(0xFFF)
    _check(gb, cuda, oracle, kt, np.ascontiguousarray(raw), 4, False)
    _check(gb, cuda, oracle, kt, np.ascontiguousarray(raw), 8, True)


@pytest.mark.parametrize("kt,ko,vo", [("u32", 1, 0), ("i32", 3, 1), ("u32", 7, 2), ("u64", 1, 3), ("i64", 3, 1)])
def test_unaligned(gb, cuda, oracle, kt, ko, vo):
    for vb in (4, 8):
        _check(gb, cuda, oracle, kt, raw_keys(kt, 40009, seed=ko), vb, True, key_offset=ko, val_offset=vo)


@pytest.mark.parametrize("kt,vb", [("u32", 4), ("u64", 8)])
def test_replayed_and_captured(gb, cuda, oracle, kt, vb):
    """The same call on a stream, replayed as a graph with other keys (uneven
    ones in the middle), and inside the caller's own capture."""
    import torch

    n = 30011
    s = torch.cuda.Stream()
    vals = np.arange(n, dtype=np.uint32 if vb == 4 else np.uint64)
    raws = [raw_keys(kt, n, seed=i) for i in range(5)]
    raws[2][:] = raws[2][0]
    raws[3][: n // 2] = raws[3][0]
    k = torch.empty(n * KEY_BYTES[kt], dtype=torch.uint8, device="cuda")
    v = torch.empty(n * vb, dtype=torch.uint8, device="cuda")
    tb = gb.temp_bytes(kt, n, vb)
    ws = torch.empty(tb, dtype=torch.uint8, device="cuda")

    def fill(raw):
        k.copy_(torch.from_numpy(raw.view(np.uint8).reshape(-1).copy()))
        v.copy_(torch.from_numpy(vals.view(np.uint8).reshape(-1).copy()))
        torch.cuda.synchronize()

    def same(raw):
        torch.cuda.synchronize()
        ek, ev = oracle.sort(kt, raw, False, vals)
        assert _eq(k.cpu().numpy().view(raw.dtype), ek) and _eq(v.cpu().numpy().view(vals.dtype), ev)

    for raw in raws:
        fill(raw)
        gb.sort(k, n, kt, ws, tb, values=v, value_bytes=vb, stream=s)
        same(raw)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        gb.sort(k, n, kt, ws, tb, values=v, value_bytes=vb, stream=torch.cuda.current_stream())
    for raw in raws:
        fill(raw)
        g.replay()
        same(raw)
