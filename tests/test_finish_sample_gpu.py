"""The sample of the sorts by leading digits (finish.cuh): arrays in order and
arrays with one heavy key look to it as they are, so that the sort stays on its
path (its outcome says so; bytes equal to the oracle's, exact: no
tolerance)."""

import numpy as np
import pytest

from _oracle import raw_keys
from test_outcome_gpu import normal, outcome_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt,n,vb", [("u64", 12_000_017, 4), ("f64", 12_000_017, 0), ("i64", 2_500_009, 8)])
def test_keys_in_order(gb, cuda, oracle, kt, n, vb):
    raw = normal(kt, n, 7) if kt == "f64" else raw_keys(kt, n, seed=7)
    raw = oracle.sort(kt, raw, False)
    assert outcome_of(gb, cuda, oracle, kt, raw, vb) == 0
    assert outcome_of(gb, cuda, oracle, kt, raw, vb, True) == 0



@pytest.mark.parametrize("kt,n", [("f64", 3_000_001), ("u64", 10_000_019)])
def test_one_heavy_key_is_no_matter(gb, cuda, oracle, kt, n):
    """One key that takes a hundredth of the array, leading bytes its own."""
    raw = normal(kt, n, 9) if kt == "f64" else raw_keys(kt, n, seed=9)
    heavy = np.random.default_rng(9).random(n) < 0.01
    if kt == "u64":
        raw[raw >> np.uint64(48) == 0] |= np.uint64(1 << 60)
        raw[heavy] = 0
    assert outcome_of(gb, cuda, oracle, kt, raw, 0 if kt == "f64" else 4) == 0
