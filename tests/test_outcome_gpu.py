"""Which path a sort took in the end (gbsort_workspace_outcome).  Every path
that is not the digit passes is followed by them on the device, so equal bytes
alone do not show that it ran: inputs that a path is for have to stay on it,
and those meant to leave it have to reach the digit passes; keys and values
equal to the oracle's all the same (exact: no tolerance).  Short key-value
arrays also in the input-preserving and DoubleBuffer forms, at the sizes where
the number of regions changes."""

import numpy as np
import pytest

from _oracle import raw_keys
from gpu_util import from_dev, to_dev

pytestmark = pytest.mark.gpu


def _eq(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


def outcome_of(gb, cuda, oracle, kt, raw, vb=0, desc=False, api="inplace"):
    """Sorts raw (with row numbers for values), checks it, returns the outcome."""
    n = raw.shape[0]
    vals = None if vb == 0 else np.arange(n, dtype=np.uint32 if vb == 4 else np.uint64)
    expect = oracle.sort(kt, raw, desc, vals)
    ek, ev = (expect, None) if vb == 0 else expect
    k = to_dev(cuda, raw)
    v = None if vb == 0 else to_dev(cuda, vals)
    both = api == "buffers"
    tb = gb.double_buffer_bytes(kt, n, vb) if both else gb.temp_bytes(kt, n, vb)
    ws = cuda.empty(tb, dtype=cuda.uint8, device="cuda")
    ws.random_(0, 256)
    if api == "inplace":
        gb.sort(k, n, kt, ws, tb, values=v, value_bytes=vb, descending=desc)
    else:
        k2, v2 = cuda.empty_like(k), None if v is None else cuda.empty_like(v)
        if both:
            if gb.sort_double_buffer(k, k2, n, kt, ws, tb, values0=v, values1=v2, value_bytes=vb, descending=desc):
                k, v = k2, v2
        else:
            gb.sort_copy(k, k2, n, kt, ws, tb, values_in=v, values_out=v2, value_bytes=vb, descending=desc)
            k, v = k2, v2
    cuda.cuda.synchronize()
    status = gb.double_buffer_status if both else gb.workspace_status
    assert status(kt, n, ws, vb) == gb.OK
    assert _eq(from_dev(k, raw), ek)
    assert vb == 0 or _eq(from_dev(v, vals), ev)
    return gb.workspace_outcome(kt, n, ws, vb, double_buffer=both)


def normal(kt, n, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal(n).astype(np.float32 if kt == "f32" else np.float64)
    x[rng.random(n) < 0.01] = -0.0
    x[:3] = [np.inf, -np.inf, np.nan]
    return x.view(np.uint32 if kt == "f32" else np.uint64)


@pytest.mark.parametrize("kt,n,vb", [
    ("u32", 3_000_001, 0), ("i64", 3_000_001, 0), ("u128", 1_500_001, 0), ("u32", 20_000_003, 0),
    ("u32", 70_001, 4), ("u64", 70_001, 8), ("u32", 1_000_003, 4), ("u64", 1_000_003, 4),
    ("u64", 2_000_003, 4), ("u128", 300_007, 8), ("i128", 50_021, 4),
])
@pytest.mark.parametrize("how", ["uniform", "ids"])
def test_stays_on_its_path(gb, cuda, oracle, kt, n, vb, how):
    raw = raw_keys(kt, n, seed=n)
    if how == "ids" and (kt.endswith("128") or n == 2_000_003):
        pytest.skip("identifiers vary in the low bytes only, which leading digits do not shorten")
    if how == "ids":
        raw = np.random.default_rng(n).integers(0, n, n).astype(raw.dtype)
    assert outcome_of(gb, cuda, oracle, kt, raw, vb) == 0


@pytest.mark.parametrize("kt,n,vb", [("f32", 9_000_001, 0), ("f64", 70_001, 0), ("f64", 3_000_001, 0), ("f64", 300_007, 4)])
def test_floats_stay_on_their_path(gb, cuda, oracle, kt, n, vb):
    assert outcome_of(gb, cuda, oracle, kt, normal(kt, n, n), vb, True) == 0


@pytest.mark.parametrize("kt,n,vb", [("u32", 3_000_001, 0), ("u64", 3_000_001, 0), ("u128", 1_500_001, 0),
                                     ("f32", 9_000_001, 0)])
def test_few_keys_take_the_digit_passes(gb, cuda, oracle, kt, n, vb):
    """Two distinct keys only: groups that no local sort takes."""
    raw = raw_keys(kt, n, seed=3)
    raw[n // 3:] = raw[0]
    raw[:n // 3] = raw[1]
    raw = raw[np.random.default_rng(1).permutation(n)]
    assert outcome_of(gb, cuda, oracle, kt, raw, vb) != 0


@pytest.mark.parametrize("kt,n,vb", [("f64", 300_007, 0), ("u64", 2_000_003, 8), ("i64", 3_000_001, 4)])
def test_low_bytes_only_take_the_digit_passes(gb, cuda, oracle, kt, n, vb):
    """Keys that vary in their low bytes: leading digits would not save a pass."""
    raw = np.random.default_rng(5).integers(0, n, n).astype(np.uint64)
    assert outcome_of(gb, cuda, oracle, kt, raw, vb) == gb.OUTCOME_PASSES


def test_key_outside_the_sampled_bits(gb, cuda, oracle):
    for kt, top in (("u32", 31), ("u64", 63)):
        raw = np.random.default_rng(2).integers(0, 1 << 16, 262_147).astype(np.uint32 if kt == "u32" else np.uint64)
        assert outcome_of(gb, cuda, oracle, kt, raw, 4) == 0
        raw[131_073] = (1 << top) + 5
        assert outcome_of(gb, cuda, oracle, kt, raw, 4) == gb.OUTCOME_PASSES


@pytest.mark.parametrize("api", ["copy", "buffers"])
@pytest.mark.parametrize("kt,vb", [("u32", 4), ("i32", 8), ("u64", 4), ("i64", 8)])
@pytest.mark.parametrize("n", [2048, 5003, 270_001, 655_001, 1_130_001])
def test_short_pairs_between_buffers(gb, cuda, oracle, api, kt, vb, n):
    assert outcome_of(gb, cuda, oracle, kt, raw_keys(kt, n, seed=n), vb, bool(n & 2), api) == 0


@pytest.mark.parametrize("api", ["copy", "buffers"])
@pytest.mark.parametrize("kt", ["u32", "u64"])
def test_short_pairs_between_buffers_fall_back(gb, cuda, oracle, api, kt):
    raw = raw_keys(kt, 262_147, seed=8)
    raw[1000:] = raw[0]
    assert outcome_of(gb, cuda, oracle, kt, raw, 4, False, api) == gb.OUTCOME_PASSES
