"""The sorts that programs using this library make, as measurable cases.

A case names an entry point (``api``), a key type, a value size, a length, an
order and a key distribution.  Lengths run from calls bound by latency to the
benchmark's largest arrays, powers of two and odd ones; distributions are the
benchmark's (uniform, N(0,1) floats with zeros, infinities and NaNs, 64-bit
keys whose upper half takes 256 values) and row identifiers below n.

Plain sorts go through the input-preserving form (the input is there again
for the next pass), or in place / between two buffers after a refill of the
buffer from its source, as a loop over fresh batches does.  Outputs are whole
buffers viewed as integers, so they compare byte for byte.
"""

from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-fast-sort_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import gbsort  # noqa: E402

_KINDS = {"u16": 2, "u32": 4, "i32": 4, "f32": 4, "u64": 8, "i64": 8, "f64": 8, "u128": 16}


def _plain(name, key, n, vb=0, dist="uniform", desc=False, api="copy"):
    c = {"api": api, "key": key, "n": n, "vb": vb, "dist": dist, "desc": desc}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a short list inside a larger program: latency only
        _plain("keys_u32_64ki", "u32", 1 << 16),
        # the benchmark's short keys-only sort
        _plain("keys_u32_1mi", "u32", 1 << 20),
        # an index built over a table of about a million rows: key and row number
        _plain("pairs_u32_1m", "u32", 1_000_003, vb=4),
        # measurements sorted in place for quantiles, batch after batch
        _plain("keys_f32_10m_inplace", "f32", 10_000_019, dist="normal", api="inplace"),
        # 64-bit hashes with a 32-bit row number: grouping and joins
        _plain("pairs_u64_u32_20m", "u64", 20_000_003, vb=4),
        # 64-bit hashes alone (distinct counts), between a caller's two buffers
        _plain("keys_u64_50m_buffers", "u64", 50_000_017, api="buffers"),
        # the benchmark's large configurations
        _plain("keys_u128_64mi_desc", "u128", 1 << 26, desc=True),
        _plain("pairs_u64_u64_128mi_desc", "u64", 1 << 27, vb=8, dist="upper256", desc=True),
        _plain("keys_u32_256mi", "u32", 1 << 28),
        _plain("pairs_f32_u32_256mi", "f32", 1 << 28, vb=4, dist="normal"),
        # the benchmark's batch: 4096 independent lists, lengths log-uniform in [2^8, 2^20]
        {"name": "batch_u32_u32_4096", "api": "batch", "key": "u32", "vb": 4, "segments": 4096, "lo": 8, "hi": 20,
         "desc": False, "dist": "uniform"},
        # the server: requests of mixed sizes from pinned host memory, submitted at once
        {"name": "served_u32_u32_24", "api": "served", "key": "u32", "vb": 4, "requests": 24, "lo": 10, "hi": 21,
         "desc": False, "dist": "uniform"},
    ]


def draw(rng):
    def log_uniform(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    r = rng.random()
    if r < 0.12:
        return {"api": "batch", "key": rng.choice(["u32", "u64"]), "vb": rng.choice([0, 4]),
                "segments": log_uniform(64, 2048), "lo": 8, "hi": rng.choice([12, 16, 20]),
                "desc": rng.random() < 0.3, "dist": "uniform"}
    if r < 0.2:
        return {"api": "served", "key": rng.choice(["u32", "f32"]), "vb": rng.choice([0, 4]),
                "requests": rng.randrange(4, 25), "lo": 10, "hi": rng.choice([16, 20, 21]), "desc": False,
                "dist": "uniform"}
    key = rng.choice(["u32", "u32", "i32", "f32", "f32", "u64", "u64", "i64", "f64", "u128", "u16"])
    vb = rng.choice([0, 0, 4, 4, 8])
    top = {2: 1 << 28, 4: 1 << 27, 8: 1 << 26, 16: 1 << 25}[_KINDS[key]]
    if key in ("f32", "f64"):
        dist = "normal"
    elif key == "u64":
        dist = rng.choice(["uniform", "uniform", "upper256", "ids"])
    elif key in ("u32", "i64"):
        dist = rng.choice(["uniform", "uniform", "ids"])
    else:
        dist = "uniform"
    return _plain("", key, log_uniform(1 << 14, top) | 1, vb, dist, rng.random() < 0.3,
                  rng.choice(["copy", "copy", "inplace", "buffers"]))


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _bits(n, g):
    """n uniform 64-bit words."""
    hi = torch.randint(0, 1 << 32, (n,), dtype=torch.int64, device="cuda", generator=g)
    return (hi << 32) | torch.randint(0, 1 << 32, (n,), dtype=torch.int64, device="cuda", generator=g)


def _keys(key, n, dist, g):
    """n keys of the type, as an integer tensor of the keys' bits."""
    kb = _KINDS[key]
    if dist == "normal":
        dt = torch.float32 if kb == 4 else torch.float64
        x = torch.randn(n, dtype=dt, device="cuda", generator=g)
        u = torch.rand(n, dtype=torch.float32, device="cuda", generator=g)
        x[u < 0.01] = -0.0
        x[(u >= 0.01) & (u < 0.0105)] = float("inf")
        x[(u >= 0.0105) & (u < 0.011)] = -float("inf")
        x[(u >= 0.011) & (u < 0.0111)] = float("nan")
        return x.view(torch.int32 if kb == 4 else torch.int64)
    if dist == "ids":
        x = torch.randint(0, n, (n,), dtype=torch.int64, device="cuda", generator=g)
        return x.to(torch.int32) if kb == 4 else x
    if dist == "upper256":
        table = torch.randint(0, 1 << 32, (256,), dtype=torch.int64, device="cuda", generator=g)
        up = table[torch.randint(0, 256, (n,), dtype=torch.int64, device="cuda", generator=g)]
        return (up << 32) | torch.randint(0, 1 << 32, (n,), dtype=torch.int64, device="cuda", generator=g)
    words = _bits((n * kb + 7) // 8, g)
    if kb >= 8:
        return words
    return words.view(torch.int16 if kb == 2 else torch.int32)[:n].clone()


def _values(vb, n):
    """Row numbers, the usual payload."""
    if not vb:
        return None
    return torch.arange(n, dtype=torch.int32 if vb == 4 else torch.int64, device="cuda")


def _lengths(case, count):
    """Log-uniform lengths in shuffled order; the case's own, whatever the
    seed, so that outputs keep their shapes."""
    lo, hi = case["lo"], case["hi"]
    r = np.random.default_rng([count, lo, hi])
    q = (np.arange(count) + r.random(count)) / count
    r.shuffle(q)
    return np.maximum(1, np.exp2(lo + (hi - lo) * q)).astype(np.int64)


def prepare(case, seed):
    g = _gen(seed)
    api, key, vb, desc = case["api"], case["key"], case["vb"], case["desc"]
    s = {"case": case, "stream": torch.cuda.current_stream()}
    if api == "batch":
        sizes = _lengths(case, case["segments"])
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
        n = int(off[-1])
        s["src"], s["vsrc"] = _keys(key, n, case["dist"], g), _values(vb, n)
        s["dst"] = torch.empty_like(s["src"])
        s["vdst"] = torch.empty_like(s["vsrc"]) if vb else None
        plan = gbsort.SegmentedPlan(key, off, vb, desc)
        s["ws"] = torch.empty(plan.workspace_bytes, dtype=torch.uint8, device="cuda")
        plan.bind(s["dst"], s["ws"], plan.workspace_bytes, values=s["vdst"], stream=s["stream"])
        s["plan"] = plan
        return s
    if api == "served":
        s["server"] = gbsort.Server(pool_bytes=1 << 30)
        reqs = []
        for n in _lengths(case, case["requests"]):
            k = _keys(key, int(n), "normal" if key == "f32" else case["dist"], g).cpu().pin_memory()
            v = _values(vb, int(n)).cpu().pin_memory() if vb else None
            reqs.append((int(n), k, v, torch.empty_like(k).pin_memory(),
                         torch.empty_like(v).pin_memory() if vb else None))
        s["reqs"] = reqs
        return s
    n = case["n"]
    s["src"], s["vsrc"] = _keys(key, n, case["dist"], g), _values(vb, n)
    s["dst"] = torch.empty_like(s["src"])
    s["vdst"] = torch.empty_like(s["vsrc"]) if vb else None
    if api == "buffers":
        s["alt"] = torch.empty_like(s["src"])
        s["valt"] = torch.empty_like(s["vsrc"]) if vb else None
        s["wsb"] = gbsort.double_buffer_bytes(key, n, vb)
    else:
        s["wsb"] = gbsort.temp_bytes(key, n, vb)
    s["ws"] = torch.empty(s["wsb"], dtype=torch.uint8, device="cuda")
    return s


def run(state):
    s, c = state, state["case"]
    api, key, vb, desc = c["api"], c["key"], c["vb"], c["desc"]
    if api == "served":
        for n, k, v, ko, vo in s["reqs"]:
            s["server"].submit(key, n, k, ko, v, vo, vb, desc)
        s["server"].drain()
        return [t for r in s["reqs"] for t in r[3:] if t is not None]
    if api == "copy":
        gbsort.sort_copy(s["src"], s["dst"], c["n"], key, s["ws"], s["wsb"], values_in=s["vsrc"],
                         values_out=s["vdst"], value_bytes=vb, descending=desc, stream=s["stream"])
    else:
        s["dst"].copy_(s["src"])
        if vb:
            s["vdst"].copy_(s["vsrc"])
    if api == "inplace":
        gbsort.sort(s["dst"], c["n"], key, s["ws"], s["wsb"], values=s["vdst"], value_bytes=vb, descending=desc,
                    stream=s["stream"])
    elif api == "batch":
        s["plan"].run(stream=s["stream"])
    elif api == "buffers":
        sel = gbsort.sort_double_buffer(s["dst"], s["alt"], c["n"], key, s["ws"], s["wsb"], values0=s["vdst"],
                                        values1=s["valt"], value_bytes=vb, descending=desc, stream=s["stream"])
        if sel:
            return [s["alt"]] + ([s["valt"]] if vb else [])
    return [s["dst"]] + ([s["vdst"]] if vb else [])


def work(case):
    """Every key and value read once and written once; a sort has no
    floating-point work."""
    kb = _KINDS[case["key"]]
    if case["api"] == "batch":
        n = int(_lengths(case, case["segments"]).sum())
    elif case["api"] == "served":
        n = int(_lengths(case, case["requests"]).sum())
    else:
        n = case["n"]
    return {"bytes": 2 * n * (kb + case["vb"]), "flops": 0}


def exact(case, seed):
    """Outputs are reordered input bits, no computed numbers."""
    return None
