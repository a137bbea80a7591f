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
