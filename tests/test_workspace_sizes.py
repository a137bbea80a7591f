"""Workspace sizes of the plain sorts: what the digit passes need is accepted by
every form, whatever shorter path the size query holds room for; that room
follows n.  (Sizes in bytes, of the in-place and input-preserving forms and of
the DoubleBuffer form.)  Host logic: an accepted call without a GPU ends as
unsupported, a refused one as too small."""

import ctypes

import numpy as np
import pytest

from _oracle import KEY_BYTES, raw_keys
from gpu_util import from_dev, to_dev

ENOUGH = [
    ("u32", 2048, 4, 28160, 11776), ("u32", 65537, 4, 557056, 32256), ("i32", 300001, 8, 3726848, 126464),
    ("u32", 1000003, 4, 8337920, 337408), ("u32", 2000003, 8, 24784384, 783872), ("u64", 2048, 8, 53760, 20992),
    ("u64", 70001, 4, 891904, 51712), ("i64", 300001, 4, 3761664, 161280), ("u64", 1000003, 4, 12492544, 492032),
    ("u128", 300007, 8, 7554304, 353792), ("f64", 70001, 0, 1457664, 897536), ("f64", 300007, 4, 3761664, 161280),
    ("f64", 3000001, 0, 25178368, 1178112), ("u32", 3000001, 4, 24992256, 991744),
]


def _calls(gb, kt, n, vb, keys, vals, keys2, vals2, ws):
    """Status of the three forms with `size` bytes of workspace."""
    l, i, sz, vp = gb.lib(), ctypes.c_int, ctypes.c_size_t, ctypes.c_void_p
    t = gb.KEY_TYPES[kt]

    def inplace(size):
        tb = sz(size)
        if vb:
            return l.gbsort_sort_pairs(t, 0, keys, vals, vb, ctypes.byref(tb), ws, n, None)
        return l.gbsort_sort_keys(t, 0, keys, ctypes.byref(tb), ws, n, None)

    def copy(size):
        try:
            gb.sort_copy(keys, keys2, n, kt, ws, size, values_in=vals, values_out=vals2, value_bytes=vb)
        except gb.GbsortError as e:
            return e.status
        return gb.OK

    def buffers(size):
        try:
            gb.sort_double_buffer(keys, keys2, n, kt, ws, size, values0=vals, values1=vals2, value_bytes=vb)
        except gb.GbsortError as e:
            return e.status
        return gb.OK

    return inplace, copy, buffers


@pytest.mark.parametrize("kt,n,vb,plain,double", ENOUGH)
def test_what_the_digit_passes_need_is_accepted(gb, kt, n, vb, plain, double):
    import torch

    if torch.cuda.is_available():
        pytest.skip("made-up addresses: without a GPU only")
    assert gb.temp_bytes(kt, n, vb) >= plain and gb.double_buffer_bytes(kt, n, vb) >= double
    inplace, copy, buffers = _calls(gb, kt, n, vb, 1 << 40, (2 << 40) if vb else None, 3 << 40,
                                    (4 << 40) if vb else None, 5 << 40)
    for call, size in ((inplace, plain), (copy, plain), (buffers, double)):
        assert call(size) == gb.ERR_UNSUPPORTED
        assert call(size - 1) == gb.ERR_WORKSPACE_TOO_SMALL


def test_room_for_regions_follows_n(gb):
    """Words of twice the key's size: at most 4.5 a pair and 8 a region for the
    DoubleBuffer form, 6 and 64 for the others."""
    for kt, n, vb, plain, double in ENOUGH:
        word = 2 * KEY_BYTES[kt]
        assert gb.temp_bytes(kt, n, vb) <= plain + (7 * n + 72 * 256) * word
        assert gb.double_buffer_bytes(kt, n, vb) <= double + (1.5 * n + 32 * 912) * word


def test_noalloc_capacity_of_doubles(gb):
    """982464 f64 keys fit the static 16 MiB, with the words of the sorts by
    leading digits."""
    import torch

    if torch.cuda.is_available():
        pytest.skip("a made-up address: without a GPU only")
    f = gb.lib().gbsort_sort_keys_noalloc
    f.restype, f.argtypes = ctypes.c_int, [ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p]
    assert f(gb.KEY_TYPES["f64"], 0, 1 << 40, 982464, None) == gb.ERR_UNSUPPORTED


@pytest.mark.gpu
@pytest.mark.parametrize("kt,n,vb,plain,double", [c for c in ENOUGH if c[1] < 1_500_000])
def test_sorts_within_them(gb, cuda, oracle, kt, n, vb, plain, double):
    """Every form sorts in exactly that much, and at sizes in between, and writes
    nothing beyond it."""
    raw = raw_keys(kt, n, seed=n)
    vals = None if not vb else np.arange(n, dtype=np.uint32 if vb == 4 else np.uint64)
    expect = oracle.sort(kt, raw, False, vals)
    ek, ev = (expect, None) if vals is None else expect
    for form, least in enumerate((plain, plain, double)):
        most = gb.double_buffer_bytes(kt, n, vb) if form == 2 else gb.temp_bytes(kt, n, vb)
        for size in sorted({least, (least + most) // 2, most}):
            ws = cuda.full((size + 4096,), 0xA5, dtype=cuda.uint8, device="cuda")
            k, k2 = to_dev(cuda, raw), cuda.empty_like(to_dev(cuda, raw))
            v = None if vals is None else to_dev(cuda, vals)
            v2 = None if v is None else cuda.empty_like(v)
            call = _calls(gb, kt, n, vb, k.data_ptr(), None if v is None else v.data_ptr(), k2.data_ptr(),
                          None if v is None else v2.data_ptr(), ws.data_ptr())[form]
            assert call(size) == gb.OK
            cuda.cuda.synchronize()
            out, vout = (k2, v2) if form == 1 else (k, v)
            assert np.array_equal(from_dev(out, raw), ek)
            assert vals is None or np.array_equal(from_dev(vout, vals), ev)
            assert bool((ws[size:] == 0xA5).all())
