"""Keys that repeat, in the sorts that work by leading bits: a crowded
sub-bucket, window or group is put in order where it is, and the sort stays on
its path (the outcome says so; bytes equal to the oracle's, exact: no
tolerance)."""

import numpy as np
import pytest

from _oracle import raw_keys
from test_outcome_gpu import outcome_of

pytestmark = pytest.mark.gpu


def repeated(kt, n, seed, copies, share=1.0):
    """A share of the keys in about `copies` copies each, the others as drawn."""
    raw = raw_keys(kt, n, seed=seed)
    rng = np.random.default_rng(seed)
    m = int(n * share)
    at = rng.permutation(n)[:m]
    raw[at] = raw[at[: max(1, m // copies)]][rng.integers(0, max(1, m // copies), m)]
    return raw


@pytest.mark.parametrize("kt,n,vb", [("u64", 3_000_001, 4), ("i64", 3_000_001, 8), ("f64", 70_001, 0),
                                     ("f64", 300_007, 4), ("u128", 300_007, 4), ("i128", 50_021, 8)])
@pytest.mark.parametrize("copies,share", [(36, 0.0005), (33, 1.0), (40, 1.0), (40, 0.5)])
def test_crowded_windows(gb, cuda, oracle, kt, n, vb, copies, share):
    assert outcome_of(gb, cuda, oracle, kt, repeated(kt, n, copies, copies, share), vb, vb == 8) == 0


@pytest.mark.parametrize("kt,n", [("u32", 3_000_001), ("i32", 20_000_003), ("u64", 3_000_001), ("i64", 30_000_001),
                                  ("u128", 1_500_001), ("i128", 1_100_003)])
@pytest.mark.parametrize("copies,share", [(33, 0.0002), (36, 0.4), (260, 0.001)])
def test_crowded_groups(gb, cuda, oracle, kt, n, copies, share):
    """Keys alone: sub-buckets of equal keys, beyond the byte counters too."""
    assert outcome_of(gb, cuda, oracle, kt, repeated(kt, n, copies, copies, share), 0, copies == 36) == 0


@pytest.mark.parametrize("kt,n", [("u32", 3_000_001), ("u64", 3_000_001), ("u128", 1_500_001)])
@pytest.mark.parametrize("size", [12, 60, 300, 520, 900])
def test_crowds_of_different_keys(gb, cuda, oracle, kt, n, size):
    """Many keys that differ in their low bits only, in one sub-bucket: put in
    order by a thread, a warp or the CTA, by their number."""
    raw = raw_keys(kt, n, seed=size)
    rng = np.random.default_rng(size)
    word = raw if kt != "u128" else raw.view(np.uint64).reshape(-1, 2)[:, 1]
    low = np.uint32(0xF) if kt == "u32" else np.uint64(0xFFFFF)
    if kt == "u128" and size > 300:
        pytest.skip("more than the groups of this many 16-byte keys have room for")
    for g in range(50):
        at = rng.integers(0, n, size)
        word[at] = (word[at] & low) | (word[at[0]] & ~low)
    assert outcome_of(gb, cuda, oracle, kt, raw) == 0


def heavy(kt, n, seed, shares):
    """A few keys of a share of the array each, among keys that share their
    leading bytes."""
    raw = raw_keys(kt, n, seed=seed)
    rng = np.random.default_rng(seed)
    draw = rng.random(n)
    at = 0.0
    for share in shares:
        raw[(draw >= at) & (draw < at + share)] = raw[rng.integers(0, n)]
        at += share
    return raw


@pytest.mark.parametrize("kt,n,vb", [("u64", 2_500_001, 4), ("i64", 9_000_011, 8), ("f64", 70_001, 4), ("f64", 600_011, 0),
                                     ("u128", 100_003, 4), ("i128", 700_001, 8)])
@pytest.mark.parametrize("shares", [(0.02,), (0.001, 0.01, 0.1), tuple([0.004] * 60), (0.45,), (0.7, 0.1)])
def test_heavy_keys(gb, cuda, oracle, kt, n, vb, shares):
    """Groups beyond a window that hold other keys too: their ranges are sorted by
    themselves, in all three forms of the call."""
    raw = heavy(kt, n, n % 97, shares)
    for api, desc in (("inplace", False), ("copy", True), ("buffers", False)):
        outcome = outcome_of(gb, cuda, oracle, kt, raw, vb, desc, api)
        assert outcome in (0, gb.OUTCOME_RANGES) or max(shares) > 0.5  # (more than half: all of it again)


def test_few_keys_of_very_many(gb, cuda, oracle):
    """Half of the array in one group of two keys: too much to take apart."""
    n = 3_000_001
    raw = raw_keys("u64", n, seed=2)
    raw[: 2 * n // 3] = 0x1234567800000000
    raw[: 2 * n // 3: 3] = 0x1234567800000001
    raw = raw[np.random.default_rng(2).permutation(n)]
    outcome_of(gb, cuda, oracle, "u64", raw, 4)
    outcome_of(gb, cuda, oracle, "u64", raw, 8, True, "copy")
    outcome_of(gb, cuda, oracle, "u64", raw, 4, False, "buffers")


@pytest.mark.parametrize("kt,n", [("u32", 3_000_001), ("i32", 12_000_017), ("u64", 2_500_001), ("i64", 26_000_003),
                                  ("u128", 1_200_007), ("i128", 5_000_011)])
@pytest.mark.parametrize("shares", [(0.01,), (0.002, 0.03, 0.1), tuple([0.003] * 50)])
def test_heavy_keys_alone(gb, cuda, oracle, kt, n, shares):
    """Groups beyond a local sort: they are sorted by themselves, in all three
    forms of the call."""
    raw = heavy(kt, n, n % 89, shares)
    for api, desc in (("inplace", False), ("copy", True), ("buffers", False)):
        assert outcome_of(gb, cuda, oracle, kt, raw, 0, desc, api) == gb.OUTCOME_RANGES
