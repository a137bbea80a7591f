"""Wide keys in order, alone, stay on the most-significant-first path (its
outcome says so; bytes equal to the oracle's, exact: no tolerance)."""

import numpy as np
import pytest

from _oracle import raw_keys
from test_outcome_gpu import outcome_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt,n", [("u64", 2_500_001), ("i64", 26_000_003), ("u128", 1_200_007), ("i128", 2_000_003)])
@pytest.mark.parametrize("desc", [False, True])
def test_wide_keys_in_order(gb, cuda, oracle, kt, n, desc):
    raw = oracle.sort(kt, raw_keys(kt, n, seed=11), False)
    assert outcome_of(gb, cuda, oracle, kt, np.ascontiguousarray(raw), 0, desc) == 0
