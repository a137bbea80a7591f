"""Key-value sorts by their leading digits (finish.cuh) at their edges: sizes
around a window, a chunk and a tile, pointers off the 16- and 32-byte
boundaries, groups of equal keys far larger than a window, groups too uneven
to finish (every digit pass then runs), leading bytes that do not vary; all
three calls, both orders, 4- and 8-byte values; keys and values equal to the
oracle's stable sort (sorts are exact: no tolerance)."""

import numpy as np
import pytest

from _oracle import KEY_BYTES, raw_keys
from gpu_util import from_dev, gpu_sort, to_dev

pytestmark = pytest.mark.gpu


def _eq(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


def _check(gb, cuda, oracle, kt, raw, vb, desc, **kw):
    vals = np.arange(raw.shape[0], dtype=np.uint32 if vb == 4 else np.uint64)
    k, v = gpu_sort(gb, cuda, kt, raw, desc, vals, **kw)
    ek, ev = oracle.sort(kt, raw, desc, vals)
    assert _eq(k, ek)
    assert _eq(v, ev)


def _spread(kt, n, seed, how):
    raw = raw_keys(kt, n, seed=seed)
    rng = np.random.default_rng(seed)
    word = raw if KEY_BYTES[kt] == 8 else raw.view(np.uint64).reshape(-1, 2)[:, 1]  # the leading 64 bits
    u = np.uint64
    if how == "spike":  # a third of the keys equal, among the others
        raw[rng.random(n) < 0.33] = raw[3]
    elif how == "all_equal":
        raw[:] = raw[3]
    elif how == "few":  # 300 distinct keys
        raw[:] = raw[:300][rng.integers(0, 300, n)]
    elif how == "runs":  # equal in all but the lowest bits, in runs of forty
        word[:] = word[rng.integers(0, max(1, n // 40), n)]
    elif how == "upper":  # 256 values of the upper half
        word[:] = (word & u(0xFFFFFFFF)) | (word[:256][rng.integers(0, 256, n)] & u(0xFFFFFFFF00000000))
    elif how == "small":  # identifiers
        word[:] = rng.integers(0, n, n).astype(np.uint64)
    elif how == "uneven":  # half of the keys in a thousandth of the range
        word[: n // 2] = (word[: n // 2] >> u(10)) + u(1 << 62)
    elif how == "sorted":
        word[:] = np.sort(word)
    return raw


@pytest.mark.parametrize("kt", ["u64", "f64", "u128", "i128"])
@pytest.mark.parametrize("n", [2047, 2048, 2875, 2876, 2877, 5001, 20000, 70001, 300007])
def test_sizes(gb, cuda, oracle, kt, n):
    for vb, desc in ((4, False), (8, True)):
        _check(gb, cuda, oracle, kt, raw_keys(kt, n, seed=n + vb), vb, desc, garbage_workspace=True)


@pytest.mark.parametrize("kt", ["u64", "i64", "u128"])
@pytest.mark.parametrize("how", ["spike", "all_equal", "few", "runs", "upper", "small", "uneven", "sorted"])
def test_spreads(gb, cuda, oracle, kt, how):
    for n, vb, desc in ((50021, 4, True), (700_001, 8, False)):
        _check(gb, cuda, oracle, kt, _spread(kt, n, n + vb, how), vb, desc)


@pytest.mark.parametrize("kt,ko,vo", [("u64", 1, 0), ("u64", 3, 1), ("f64", 2, 3), ("u128", 1, 1), ("i64", 0, 5)])
def test_unaligned(gb, cuda, oracle, kt, ko, vo):
    for vb in (4, 8):
        _check(gb, cuda, oracle, kt, raw_keys(kt, 40009, seed=ko), vb, False, key_offset=ko, val_offset=vo)


@pytest.mark.parametrize("kt", ["u64", "f128"])
@pytest.mark.parametrize("how", ["plain", "uneven", "small"])
def test_input_preserving_and_double_buffer(gb, cuda, oracle, kt, how):
    n = 90_001
    raw = _spread(kt, n, 9, how)
    vals = np.arange(n, dtype=np.uint32)
    ek, ev = oracle.sort(kt, raw, True, vals)
    src, vsrc = to_dev(cuda, raw), to_dev(cuda, vals)
    out, vout = cuda.zeros_like(src), cuda.zeros_like(vsrc)
    tb = gb.temp_bytes(kt, n, 4)
    ws = cuda.empty(tb, dtype=cuda.uint8, device="cuda")
    gb.sort_copy(src, out, n, kt, ws, tb, values_in=vsrc, values_out=vout, value_bytes=4, descending=True)
    cuda.cuda.synchronize()
    assert gb.workspace_status(kt, n, ws, 4) == gb.OK
    assert _eq(from_dev(out, raw), ek) and _eq(from_dev(vout, vals), ev)
    assert _eq(from_dev(src, raw), raw) and _eq(from_dev(vsrc, vals), vals)
    dbb = gb.double_buffer_bytes(kt, n, 4)
    dws = cuda.empty(dbb, dtype=cuda.uint8, device="cuda")
    k0, v0 = cuda.zeros_like(src), cuda.zeros_like(vsrc)
    sel = gb.sort_double_buffer(k0, src, n, kt, dws, dbb, selector=1, values0=v0, values1=vsrc, value_bytes=4,
                                descending=True)
    cuda.cuda.synchronize()
    assert gb.double_buffer_status(kt, n, dws, 4) == gb.OK
    assert _eq(from_dev(src if sel else k0, raw), ek) and _eq(from_dev(vsrc if sel else v0, vals), ev)


@pytest.mark.parametrize("n", [16383, 16384, 70001, 300007, (1 << 21) + 1])
@pytest.mark.parametrize("how", ["normal", "spike", "uneven", "few"])
def test_floats_without_values(gb, cuda, oracle, n, how):
    if how == "normal":
        rng = np.random.default_rng(n)
        x = rng.standard_normal(n)
        x[rng.random(n) < 0.02] = -0.0
        x[:5] = [np.inf, -np.inf, np.nan, 0.0, 5e-324]
        raw = x.view(np.uint64)
    else:
        raw = _spread("f64", n, n, how)
    for desc in (False, True):
        assert _eq(gpu_sort(gb, cuda, "f64", raw, desc, garbage_workspace=True, key_offset=1), oracle.sort("f64", raw, desc))
