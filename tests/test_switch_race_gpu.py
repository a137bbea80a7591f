"""A switch changed by another thread while sorts are queued: every sort is
planned, launched and cached under one reading of it, so its result is the
oracle's either way (exact: no tolerance).  Key-value floats make their digit
passes in one launch, whose buffers depend on pass skipping."""

import ctypes
import threading

import numpy as np
import pytest

from _oracle import raw_keys
from gpu_util import to_dev

pytestmark = pytest.mark.gpu


def test_pass_skip_toggled_while_sorting(gb, cuda, oracle):
    n, rounds = 3001, 3000
    raw = raw_keys("f64", n, seed=4)
    vals = np.arange(n, dtype=np.uint32)
    ek, ev = oracle.sort("f64", raw, False, vals)
    src, vsrc, ek, ev = to_dev(cuda, raw), to_dev(cuda, vals), to_dev(cuda, ek), to_dev(cuda, ev)
    k, v = cuda.empty_like(src), cuda.empty_like(vsrc)
    tb = gb.temp_bytes("f64", n, 4)
    ws = cuda.empty(tb, dtype=cuda.uint8, device="cuda")
    wrong = cuda.zeros(1, dtype=cuda.int64, device="cuda")
    stop = threading.Event()
    toggle = ctypes.CDLL(gb.LIB_PATH).gbsort_set_pass_skip

    def switch():
        while not stop.is_set():
            for on in (0, 1) * 50:
                toggle(on)

    t = threading.Thread(target=switch)
    t.start()
    try:
        for _ in range(rounds):
            k.copy_(src)
            v.copy_(vsrc)
            gb.sort(k, n, "f64", ws, tb, values=v, value_bytes=4)
            wrong += (k != ek).any() | (v != ev).any()
        cuda.cuda.synchronize()
    finally:
        stop.set()
        t.join()
        gb.set_pass_skip(True)
    assert int(wrong) == 0
