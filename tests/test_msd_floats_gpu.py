"""Keys-only sorts of 4-byte floats most significant bits first (msd.cuh):
group numbers from the sample's distribution, groups of equal keys above and
below the largest that a local sort takes, values that the sample may miss,
ranges that end inside a bin, tiles whose digits overflow their places; every
result equal to the oracle's bytes (sorts are exact: no tolerance)."""

import numpy as np
import pytest

from _oracle import raw_keys
from gpu_util import gpu_sort

pytestmark = pytest.mark.gpu

LEAST = 1 << 23  # the path's smallest array


def _eq(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


def _values(dist, n, rng):
    x = rng.standard_normal(n, dtype=np.float32)
    if dist == "special":
        u = rng.random(n, dtype=np.float32)
        for lo, hi, v in ((0.0, 0.2, 0.0), (0.2, 0.21, -0.0), (0.21, 0.22, np.inf), (0.22, 0.221, -np.inf),
                          (0.221, 0.2212, np.nan), (0.2212, 0.22121, 3e38)):
            x[(u >= lo) & (u < hi)] = v
    elif dist == "to_900":
        x = rng.random(n, dtype=np.float32) * np.float32(900)
    elif dist == "one_exponent":
        x = rng.random(n, dtype=np.float32) + np.float32(1)
    elif dist == "outliers":  # outside the range that the sample's keys share
        x = rng.random(n, dtype=np.float32) + np.float32(1)
        for i, v in enumerate((0.0, -0.0, -5.0, 1e30, np.inf, 0.25, 64.0)):
            x[rng.integers(0, n, 1 + 3 * i)] = v
    elif dist == "exponential":
        x = rng.standard_exponential(n, dtype=np.float32)
    elif dist == "rounded":  # few values: too crowded for the local sorts
        x = np.round(x * 64)
    elif dist == "mixed_giant":  # one bin: nearly all equal, but not all
        x[rng.random(n, dtype=np.float32) < 0.02] = 3e-30
        x[:: n // 7] = 3.1e-30
        x[1 :: n // 5] = 2.9e-30
    elif dist == "many_giants":  # more large groups of equal keys than the list holds
        u = rng.integers(0, 100, n)
        x = np.where(u < 60, np.ldexp(np.float32(1), -100 + u).astype(np.float32), x)
    elif dist == "crowds":  # values that the sample misses, 40 to 600 times each
        for i, c in enumerate((33, 40, 64, 255, 256, 300, 600)):
            x[rng.integers(0, n, c)] = np.float32(1.5 + i * 0.01)
    return x.view(np.uint32)


@pytest.mark.parametrize("desc", [False, True])
@pytest.mark.parametrize("dist", ["normal", "special", "to_900", "one_exponent", "outliers", "exponential",
                                  "rounded", "mixed_giant", "many_giants", "crowds"])
def test_distributions(gb, cuda, oracle, dist, desc):
    rng = np.random.default_rng(len(dist) + desc)
    raw = _values(dist, LEAST + 4099, rng).astype(raw_keys("f32", 1, 0).dtype)
    assert _eq(gpu_sort(gb, cuda, "f32", raw, desc, key_offset=int(desc)), oracle.sort("f32", raw, desc))


@pytest.mark.parametrize("n,offset", [(LEAST - 1, 0), (LEAST, 1), (LEAST + 1, 2), (11796481, 3), (23592961, 0)])
def test_sizes(gb, cuda, oracle, n, offset):
    raw = _values("special", n, np.random.default_rng(n)).astype(raw_keys("f32", 1, 0).dtype)
    assert _eq(gpu_sort(gb, cuda, "f32", raw, False, key_offset=offset), oracle.sort("f32", raw, False))


def test_random_bits_and_sorted(gb, cuda, oracle):
    raw = raw_keys("f32", LEAST + 77, seed=3)
    want = oracle.sort("f32", raw, False)
    assert _eq(gpu_sort(gb, cuda, "f32", raw, False), want)
    assert _eq(gpu_sort(gb, cuda, "f32", want, False), want)
