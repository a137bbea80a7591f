"""gbsort_route (host logic): the path of a sort by type, values and size, the
launches that it makes, what the timed entry point runs instead, and the
workspace sizes that the queries give."""

import pytest


@pytest.mark.parametrize("kt,n,vb,path,launches,timed", [
    ("u32", 1 << 20, 0, "ONE_LAUNCH", 1, "ONE_LAUNCH"), ("u32", 1 << 26, 0, "MSD", 8, "MSD"),
    ("f32", 1 << 24, 0, "MSD", 8, "MSD"), ("f32", 5_000_000, 0, "PASSES", 6, "PASSES"),
    ("u128", 1 << 24, 0, "MSD", 8, "MSD"), ("f64", 1 << 20, 0, "LEADING_DIGITS", 6, "ONE_LAUNCH"),
    ("f64", 1 << 25, 0, "LEADING_DIGITS", 6, "MSD"), ("u32", 1 << 20, 4, "SHORT_PAIRS", 2, "PASSES"),
    ("u64", 1_000_003, 8, "SHORT_PAIRS", 2, "PASSES"), ("u64", 1 << 24, 4, "LEADING_DIGITS", 6, "PASSES"),
    ("u32", 1 << 24, 4, "PASSES", 6, "PASSES"), ("u32", 1 << 24, 2, "PASSES", 6, "PASSES"),
    ("u16", 1 << 24, 0, "PASSES", 4, "PASSES"), ("u128", 1 << 20, 4, "LEADING_DIGITS", 6, "PASSES"),
])
def test_paths(gb, kt, n, vb, path, launches, timed):
    r = gb.route(kt, n, vb)
    assert (r.path, r.kernel_launches) == (getattr(gb, "PATH_" + path), launches)
    assert r.timed_path == getattr(gb, "PATH_" + timed)
    assert r.workspace_bytes == gb.temp_bytes(kt, n, vb) >= r.workspace_min_bytes
    assert r.double_buffer_bytes == gb.double_buffer_bytes(kt, n, vb) >= r.double_buffer_min_bytes


def test_switches_change_the_path_not_the_sizes(gb):
    before = {c: gb.route(*c) for c in (("u64", 1_000_003, 4), ("u64", 1 << 24, 4), ("u32", 1 << 26, 0))}
    gb.set_pass_skip(False)
    gb.set_msd(False)
    try:
        for c, b in before.items():
            r = gb.route(*c)
            assert r.path == gb.PATH_PASSES and r.workspace_bytes == b.workspace_bytes
            assert r.kernel_launches == gb.plan(*c).kernel_launches == gb.plan(*c).passes + 1
    finally:
        gb.set_pass_skip(True)
        gb.set_msd(True)


def test_each_path_of_pairs_alone(gb):
    """Short pairs and leading digits switch off one by one; sizes stay."""
    short, wide = ("u64", 1_000_003, 4), ("u64", 1 << 24, 4)
    sizes = [gb.temp_bytes(*c) for c in (short, wide)]
    assert gb.short_pairs() and gb.leading_digits()
    try:
        gb.short_pairs(False)
        assert gb.route(*short).path == gb.PATH_LEADING_DIGITS and gb.route(*wide).path == gb.PATH_LEADING_DIGITS
        gb.leading_digits(False)
        assert gb.route(*short).path == gb.route(*wide).path == gb.PATH_PASSES
        gb.short_pairs(True)
        assert gb.route(*short).path == gb.PATH_SHORT_PAIRS
        assert [gb.temp_bytes(*c) for c in (short, wide)] == sizes
    finally:
        gb.short_pairs(True)
        gb.leading_digits(True)


@pytest.mark.gpu
def test_switched_off_they_sort_the_same(gb, cuda, oracle):
    from _oracle import raw_keys
    from test_outcome_gpu import outcome_of

    for short, wide in ((False, True), (True, False), (False, False)):
        gb.short_pairs(short)
        gb.leading_digits(wide)
        try:
            for kt, n, vb in (("u32", 70_001, 4), ("u64", 300_007, 8), ("f64", 20_001, 0), ("u128", 20_001, 4)):
                outcome_of(gb, cuda, oracle, kt, raw_keys(kt, n, seed=1), vb, True)
        finally:
            gb.short_pairs(True)
            gb.leading_digits(True)
