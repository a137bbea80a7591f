"""Keys-only sorts most significant bits first where groups, sub-buckets and
tiles are at their edges (msd.cuh): sizes around the lower end of the path
and where the number of groups doubles, pointers off the 16- and 32-byte
boundaries, counters that pass 2^15 and 255, sub-buckets beyond the network's
margin and beyond the comparison rank; every result equal to the oracle's
bytes (sorts are exact: no tolerance)."""

import numpy as np
import pytest

from _oracle import KEY_BYTES, raw_keys
from gpu_util import gpu_sort

pytestmark = pytest.mark.gpu


def _eq(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


@pytest.mark.parametrize("kt,n,offset", [
    ("u32", (1 << 21) + 1, 0), ("i32", (1 << 21) + 1, 1), ("f32", 4194303, 2), ("u32", (1 << 22) + 1, 3),
    ("u32", 8481792, 5), ("f32", 8481793, 7), ("i32", 5000011, 4),
    ("u64", (1 << 21) + 1, 1), ("f64", 4240897, 2), ("i64", (1 << 22) + 3, 3),
    ("u128", (1 << 20) + 1, 1), ("f128", (3 << 19) - 1, 0),
])
@pytest.mark.parametrize("desc", [False, True])
def test_sizes_and_alignment(gb, cuda, oracle, kt, n, offset, desc):
    raw = raw_keys(kt, n, seed=n % 1000 + int(desc))
    assert _eq(gpu_sort(gb, cuda, kt, raw, desc, key_offset=offset), oracle.sort(kt, raw, desc))


@pytest.mark.parametrize("kt", ["u32", "u64"])
@pytest.mark.parametrize("crowd", [9, 17, 32, 33, 255, 256, 600])
def test_crowded_sub_buckets(gb, cuda, oracle, kt, crowd):
    """`crowd` keys that share all but their low bits, in many groups."""
    n = 3_000_001
    raw = raw_keys(kt, n, seed=crowd)
    bits = 8 * KEY_BYTES[kt]
    low = raw.dtype.type((1 << (3 if kt == "u32" else 32)) - 1)
    rng = np.random.default_rng(crowd)
    for g in range(40):
        at = rng.integers(0, n - crowd)
        base = raw.dtype.type((g * 6 + 1) << (bits - 8)) | (raw[at] & raw.dtype.type((1 << (bits - 9)) - 1) & ~low)
        raw[at:at + crowd] = (raw[at:at + crowd] & low) | base
    assert _eq(gpu_sort(gb, cuda, kt, raw, False), oracle.sort(kt, raw, False))


@pytest.mark.parametrize("kt", ["u32", "f64"])
@pytest.mark.parametrize("share", [0.001, 0.3, 1.0])
def test_repeated_keys_and_one_group(gb, cuda, oracle, kt, share):
    """A share of the keys equal (a group counter past 2^15), and keys whose
    leading bits take three values only."""
    n = 6_000_007
    raw = raw_keys(kt, n, seed=5)
    raw[: int(n * share)] = raw[1]
    rng = np.random.default_rng(1)
    raw = raw[rng.permutation(n)]
    assert _eq(gpu_sort(gb, cuda, kt, raw, True), oracle.sort(kt, raw, True))
    bits = 8 * KEY_BYTES[kt]
    few = raw & raw.dtype.type((1 << (bits - 16)) - 1)
    few |= rng.integers(0, 3, n).astype(raw.dtype) << raw.dtype.type(bits - 2)
    assert _eq(gpu_sort(gb, cuda, kt, few, False), oracle.sort(kt, few, False))
