"""The verify path's performance cases: what a user of this package has it do,
each through its public entry points (goldbach-l0_gb300/gbc.py over
include/gbc.h), from one small window to production slices.

A case is a dict of plain values; its "kind" names the entry point:

  range    Context.verify_range: a run of consecutive evens (the whole of
           gb::run_gpu), p(n) of every even or production sampling, with or
           without the per-even p(n) array
  segment  Context.enqueue_batch + Context.collect: the per-segment contract,
           one production segment per batch
  windows  Context.verify_windows: many windows of uneven widths and heights
           in shared batches
  serve    Server.submit + Server.wait: windows handed to the serving loop
           together, each waited for
  sparse   Sparse.verify: the sparse class map cross-check
  noalloc  gbc_class_map_noalloc: the class map of a range of q into the
           caller's own buffer

What a program has in hand before the call is a context made once for all of
its ranges (sieving primes, slots, the prime-multiplier table built ahead):
states of one configuration share it, as the ranges of one program do. The
last one made stays open; the one before is closed with its last state.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "goldbach-l0_gb300"))
import gbc  # noqa: E402

SEG = gbc.DEFAULT_SEGMENT
SLICE = 4 * 10**18                  # the production slices start here
LINE = 1 << 16                      # bytes of a run's statistics line, zero-padded
U30 = (1, 7, 11, 13, 17, 19, 23, 29)

# the sieve and plan knobs of tuning/gb300_production_4e18.json ("" leaves
# every knob at the library's default)
KNOBS = {"": {}, "tuned": {"p_mid": 1703936, "mtab_max_gb": 160, "tile_bits": 1835008, "plan_funnels": 16,
                           "verify_funnels": 3}}


def listed():
    none = gbc.SAMPLE_NONE
    return [
        # production: two batches of 128 segments with the recorded knobs, every
        # 256th segment p(n) of every even, the others the funnel verify
        {"name": "slice", "kind": "range", "height": float(SLICE), "width": 256 * SEG, "batch": 128,
         "knobs": "tuned", "sample": 256, "pn": False},
        # the same with p(n) of every even on every segment (the exact statistics)
        {"name": "slice_exact", "kind": "range", "height": float(SLICE), "width": 48 * SEG, "batch": 48,
         "knobs": "tuned", "sample": 1, "pn": False},
        # a short slice by a user who sets no knobs: eight segments per batch
        {"name": "slice_default", "kind": "range", "height": float(SLICE), "width": 24 * SEG + 40_000_010, "batch": 8,
         "knobs": "", "sample": 256, "pn": False},
        # the reference's own unit: one 467.5M segment through enqueue and collect
        {"name": "segment", "kind": "segment", "height": float(SLICE), "width": SEG, "batch": 8, "knobs": "",
         "sample": 256},
        # the plain window at 1e12: 5e8 evens, tile primes only, exact statistics
        {"name": "range_1e12", "kind": "range", "height": 1e12, "width": 1_000_000_000, "batch": 8, "knobs": "",
         "sample": 1, "pn": False},
        # p(n) of every even handed back, an odd width
        {"name": "range_pn", "kind": "range", "height": 1e12, "width": 20_000_002, "batch": 8, "knobs": "",
         "sample": 1, "pn": True},
        # the smallest call: half a million evens, where launches and latency count
        {"name": "range_small", "kind": "range", "height": 1e12, "width": 1_000_000, "batch": 8, "knobs": "",
         "sample": 1, "pn": False},
        # uneven windows, widths log-uniform in [1e6, 1e10], starts in [1e15, 5e18]:
        # p(n) of every even, and verification without sampling
        {"name": "windows_exact", "kind": "windows", "count": 64, "lo": 1e6, "hi": 1e10, "low": 1e15, "high": 5e18,
         "knobs": "tuned", "sample": 1},
        {"name": "windows_verify", "kind": "windows", "count": 96, "lo": 1e6, "hi": 1e10, "low": 1e15, "high": 5e18,
         "knobs": "tuned", "sample": none},
        # a burst of requests at the serving loop: widths in [1e4, 1e9], starts in [1e10, 5e18]
        {"name": "serve", "kind": "serve", "count": 32, "lo": 1e4, "hi": 1e9, "low": 1e10, "high": 5e18,
         "knobs": "tuned"},
        # the independent cross-check: one segment of 30030 * 2^26 integers and a ragged end
        {"name": "sparse", "kind": "sparse", "height": float(SLICE), "dlt_log2": 26, "width": 2_100_000_000_002},
        # a class map of 2^29 integers for a caller that cannot allocate
        {"name": "noalloc", "kind": "noalloc", "height": 1e12, "width": 1 << 29},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("range", "range", "low", "segment", "windows", "windows", "serve", "sparse", "noalloc"))
    knobs = rng.choice(("", "tuned"))
    sample = rng.choice((1, 256, gbc.SAMPLE_NONE))
    if kind == "low":  # from the first evens on: the generic low checker and small q
        return {"kind": "range", "height": 4.0, "width": int(_log(rng, 1e5, 1e9)) // 2 * 2, "batch": 8, "knobs": "",
                "sample": 1, "pn": rng.random() < 0.3}
    if kind == "range":
        height = rng.choice((float(SLICE), _log(rng, 1e10, 5e18)))
        pn = rng.random() < 0.25
        width = _log(rng, 1e6, 1e8 if pn else 96 * SEG if sample == 1 else 192 * SEG)
        # slots for the run: as many production segments as it holds, up to 128
        batch = 8 if not knobs else min(128, max(8, int(width) // SEG + 1))
        return {"kind": kind, "height": height, "width": int(width) // 2 * 2, "batch": batch,
                "knobs": "" if pn else knobs, "sample": 1 if pn else sample, "pn": pn}
    if kind == "segment":
        return {"kind": kind, "height": _log(rng, 1e15, 5e18), "width": int(_log(rng, 1e7, SEG)) // 2 * 2, "batch": 8,
                "knobs": knobs, "sample": rng.choice((1, 256))}
    if kind == "windows":
        lo = _log(rng, 1e6, 1e8)
        return {"kind": kind, "count": int(_log(rng, 8, 96)), "lo": lo, "hi": min(1e10, lo * _log(rng, 10, 1e4)),
                "low": 1e15, "high": 5e18, "knobs": "tuned", "sample": rng.choice((1, gbc.SAMPLE_NONE))}
    if kind == "serve":
        lo = _log(rng, 1e4, 1e7)
        return {"kind": kind, "count": int(_log(rng, 1, 64)), "lo": lo, "hi": min(1e9, lo * _log(rng, 10, 1e5)),
                "low": 1e10, "high": 5e18, "knobs": "tuned"}
    if kind == "sparse":
        dlt = rng.randint(16, 25)
        return {"kind": kind, "height": _log(rng, 1e15, 5e18), "dlt_log2": dlt,
                "width": int(30030 * 2**dlt * _log(rng, 0.3, 1.9)) // 2 * 2}
    return {"kind": kind, "height": _log(rng, 1e8, 2.9e12), "width": int(_log(rng, 1e5, 1 << 30))}


# ---- what a program keeps between calls ------------------------------------------

class _Held:
    """A context (with a server over it) or a Sparse, closed with its last user."""

    def __init__(self, make):
        self.server = None
        self.obj = make()

    def __del__(self):
        if self.server is not None:
            self.server.stop()
        if getattr(self, "obj", None) is not None:
            self.obj.close()


_last = {}


def _hold(key, make):
    if key not in _last:
        _last.clear()
        _last[key] = make()
    return _last[key]


def _top(case):
    """The largest even any seed of the case reaches."""
    if case["kind"] in ("windows", "serve"):
        return int(case["high"] + case["hi"]) // 2 * 2 + 2
    if case["kind"] == "range" and case["height"] < 100:
        return case["width"] + 1000
    return _floor(case) + _spread(case) + case["width"] + 2


def _floor(case):
    return int(case["height"]) // 2 * 2


def _spread(case):
    """How far the seeds move a start: over the 5e13 slice at production height, 2% of the height elsewhere."""
    return 5 * 10**13 if case["height"] >= 1e15 else int(case["height"]) // 50


def _start(case, rng):
    if case["height"] < 100:
        return 4
    step = SEG if case["height"] == SLICE else 2
    return _floor(case) + rng.randrange(_spread(case) // step) * step


def _context(case):
    kind, knobs = case["kind"], KNOBS[case["knobs"]]
    top = _top(case)
    shape = {"range": lambda: {"max_batch": case["batch"], "want_pn": case["pn"], "sample_every": case["sample"]},
             "segment": lambda: {"max_batch": case["batch"]},
             "windows": lambda: {"max_batch": 64, "max_runs": 64, "nslots": 3, "sample_every": case["sample"]},
             "serve": lambda: {"max_batch": 16, "max_runs": 16, "nslots": 4}}[kind]()

    def make():
        # a run shorter than a segment with the p(n) array: slots no wider than it
        seg = min(SEG, (case["width"] + 2000) // 1000 * 1000) if shape.get("want_pn") else SEG
        held = _Held(lambda: gbc.Context(limit=top, segment_even=seg, **shape, **knobs))
        if kind == "serve":
            held.server = gbc.Server(held.obj, hbm_budget=150 * 10**9, lo=int(case["low"]), hi=top)
        elif case.get("low", case.get("height")) > 1e6:
            held.obj.prepare(int(case.get("low", case.get("height"))) // 2 * 2, top)
        return held

    return _hold((kind, top, case["knobs"], tuple(sorted(shape.items())),
                  case["width"] if shape.get("want_pn") else 0), make)


def _windows(case, rng):
    """Windows with widths spread evenly over the logarithm of [lo, hi], in random order."""
    n, lo, hi = case["count"], math.log(case["lo"]), math.log(case["hi"])
    widths = [int(math.exp(lo + (hi - lo) * (i + rng.random()) / n)) // 2 * 2 for i in range(n)]
    rng.shuffle(widths)
    wins = []
    for w in widths:
        a = _log(rng, case["low"], case["high"]) if case["kind"] == "serve" else rng.uniform(case["low"], case["high"])
        wins.append((int(a) // 2 * 2, int(a) // 2 * 2 + w))
    return wins


def prepare(case, seed):
    rng = random.Random("%s %d" % (case["kind"], seed))
    kind = case["kind"]
    state = {"case": case}
    if kind == "sparse":
        top = _top(case)
        state["held"] = _hold(("sparse", top, case["dlt_log2"]),
                              lambda: _Held(lambda: gbc.Sparse(limit=top, dlt_log2=case["dlt_log2"])))
        a = _start(case, rng)
        state["range"] = (a, a + case["width"] - 2)
        return state
    if kind == "noalloc":
        a = int(case["height"]) + rng.randrange(int(case["height"]) // 50)
        primes = _odd_primes(math.isqrt(a + case["width"]) + 400)  # the last one at or above the root
        lib, wpc = gbc.load(), ctypes.c_uint32()
        dev = torch.from_numpy(primes.astype(np.int32)).cuda()
        lib.gbc_class_map_noalloc(a, a + case["width"] - 1, dev.data_ptr(), len(primes), int(primes[-1]), None, 0,
                                  None, None, ctypes.byref(wpc), None, None, 0)  # the size of the map
        state.update(range=(a, a + case["width"] - 1), primes=dev, max_prime=int(primes[-1]),
                     map=torch.zeros(8 * wpc.value, dtype=torch.int32, device="cuda"))
        return state
    state["held"] = _context(case)
    if kind in ("windows", "serve"):
        state["windows"] = _windows(case, rng)
        return state
    a = _start(case, rng)
    w = case["width"]
    if case["height"] < 100:  # a run from the first evens on ends where the seed says
        w -= 2 * rng.randrange(w // 200)
    state["range"] = (a, a + w - 2)
    return state


def _line(text):
    return np.frombuffer(text.encode().ljust(LINE, b"\0"), dtype=np.uint8)


def _counts(r):
    return [r.evens, r.segments, r.leftovers, r.pmax, r.primes, r.twins]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "range":
        ctx, (a, b) = state["held"].obj, state["range"]
        res, line, pn = ctx.verify_range(a, b, want_pn=case["pn"])
        out = {"counts": np.array(_counts(res), dtype=np.int64), "line": _line(line)}
        if pn is not None and case["height"] >= 100:
            out["pn"] = np.frombuffer(pn, dtype=np.int16)
        elif pn is not None:  # the run's length differs from seed to seed
            out["pn"] = np.frombuffer(pn, dtype=np.int16)[:(case["width"] - case["width"] // 100) // 2 - 2]
        return out
    if kind == "segment":
        ctx, (a, b) = state["held"].obj, state["range"]
        ctx.enqueue_batch(0, [(a, b)], b, [0 if case["sample"] == 1 else gbc.SEG_VERIFY])
        (s,), _ = ctx.collect(0, 1)
        tails = np.zeros(gbc.TAIL_CAP, dtype=np.uint64)
        tails[:s.ntail] = np.sort(np.frombuffer(s.tail_lo, dtype=np.uint64)[:s.ntail])
        ridges = np.zeros(gbc.RIDGE_CAP, dtype=np.uint64)
        ridges[:s.nridge] = np.sort(np.frombuffer(s.ridge_n, dtype=np.uint64)[:s.nridge])
        words = np.array([s.evens, s.map_hash, s.map_primes, s.gmax_key, s.first_prime, s.last_prime, s.pending,
                          s.nleft, s.ntail, s.nridge], dtype=np.uint64)
        return {"words": words.view(np.int64), "hist": np.frombuffer(s.hist, dtype=np.int32),
                "first": np.frombuffer(s.first, dtype=np.int32), "ghist": np.frombuffer(s.ghist, dtype=np.int32),
                "primes30": np.frombuffer(s.primes30, dtype=np.int64),
                "twins": np.frombuffer(s.twins, dtype=np.int64),
                "tails": tails.view(np.int64), "ridges": ridges.view(np.int64)}
    if kind == "windows":
        got, _ = state["held"].obj.verify_windows(state["windows"])
        return {"counts": np.array([_counts(r) for r, _ in got], dtype=np.int64),
                "lines": np.concatenate([_line(t) for _, t in got])}
    if kind == "serve":
        srv = state["held"].server
        tickets = [srv.submit(a, b) for a, b in state["windows"]]
        got = [srv.wait(t) for t in tickets]
        return {"counts": np.array([_counts(r) for r, _, _ in got], dtype=np.int64),
                "lines": np.concatenate([_line(t) for _, t, _ in got])}
    if kind == "sparse":
        sp, (a, b) = state["held"].obj, state["range"]
        r = sp.verify(a, b)
        return {"counts": np.array([r.evens, r.pending, r.map_primes, r.segments], dtype=np.int64)}
    a, b = state["range"]
    primes, m = state["primes"], state["map"]
    base, nblk, wpc = ctypes.c_uint64(), ctypes.c_uint32(), ctypes.c_uint32()
    err = ctypes.create_string_buffer(256)
    rc = gbc.load().gbc_class_map_noalloc(a, b, primes.data_ptr(), primes.numel(), state["max_prime"], m.data_ptr(),
                                          m.numel(), ctypes.byref(base), ctypes.byref(nblk), ctypes.byref(wpc),
                                          torch.cuda.current_stream().cuda_stream, err, len(err))
    if rc:
        raise gbc.GbcError(rc, err.value.decode())
    return {"map": m, "layout": np.array([base.value - a, nblk.value - case["width"] // 30], dtype=np.int64)}


def work(case):
    """Bytes: the sieving primes up to the root of the top read once, the class
    map (8 bits per 30 integers; 12 classes mod 30030 on the sparse path) written
    and read once, the results written. Operations: the multiples of the primes
    from 71 on cleared in the map, and one candidate test per even."""
    if case["kind"] in ("windows", "serve"):
        n = case["count"]
        span = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"]) * n  # the log-uniform mean
        top = case["high"]
    elif case["kind"] == "sparse":
        n, span, top = 1, float(case["width"]), case["height"]
    else:
        n, span, top = 1, float(case["width"]), max(case["height"], float(case["width"]))
    root = math.sqrt(top)
    primes = 4 * root / max(1.0, math.log(root) - 1)
    classes, mod = (12, 30030) if case["kind"] == "sparse" else (8, 30)
    bits = span * classes / mod
    marks = bits * math.log(math.log(max(root, 80)) / math.log(71))
    if case["kind"] == "noalloc":
        return {"bytes": primes + bits / 8, "flops": marks}
    out = span / 2 * (2 if case.get("pn") else 0) + n * 8192
    return {"bytes": primes + 2 * bits / 8 + out, "flops": marks + span / 2}


# ---- the same results by plain numpy ----------------------------------------------

def _odd_primes(n):
    s = np.ones(n + 1, dtype=bool)
    s[:2] = False
    s[4::2] = False
    for i in range(3, math.isqrt(n) + 1, 2):
        if s[i]:
            s[i * i::i] = False
    p = np.nonzero(s)[0]
    return p[p > 2].astype(np.int64)


def _sieve(lo, hi):
    """is[q - lo] for q in [lo, hi], lo even: primality by a segmented sieve."""
    s = np.ones(hi - lo + 1, dtype=bool)
    s[0::2] = False
    for p in _odd_primes(math.isqrt(hi) + 1).tolist():
        s[max(p * p, (lo + p - 1) // p * p) - lo::p] = False
    if lo <= 2:
        s[2 - lo] = True
    if lo <= 1:
        s[:2 - lo] = False
    return s


def exact(case, seed):
    rng = random.Random("%s %d" % (case["kind"], seed))
    if case["kind"] == "noalloc" and case["width"] <= 1 << 29:
        a = int(case["height"]) + rng.randrange(int(case["height"]) // 50)
        b = a + case["width"] - 1
        base, nblk = a // 30 * 30, (b - a // 30 * 30) // 30 + 1
        wpc = (nblk + 64 + 65535) // 65536 * 2048
        s = _sieve(base, base + 30 * nblk)
        out = np.zeros((8, 4 * wpc), dtype=np.uint8)
        for k, u in enumerate(U30):
            bits = np.packbits(s[u:30 * nblk:30], bitorder="little")
            out[k, :len(bits)] = bits
        return {"map": out.reshape(-1).view(np.int32), "layout": np.array([base - a, nblk - case["width"] // 30])}
    if case["kind"] == "range" and 1e4 <= case["height"] <= 1e13 and case["width"] <= 3e7:
        a = _start(case, rng)
        b = a + case["width"] - 2
        lo = a - 10000
        s = _sieve(lo, b + 2)
        n = np.arange(a, b + 1, 2) - lo
        pn = np.zeros(len(n), dtype=np.int16)
        open_ = np.arange(len(n))
        for p in _odd_primes(9800).tolist():
            hit = s[n[open_] - p]
            pn[open_[hit]] = p
            open_ = open_[~hit]
            if not len(open_):
                break
        if len(open_):
            return None
        # primes in [a + 1, b - 1] and twins (q, q + 2) inside it
        c = s[a + 1 - lo:b - lo]
        twins = int(np.count_nonzero(c[:-2] & c[2:]))
        segments = -(-case["width"] // (SEG if not case["pn"] else (case["width"] + 2000) // 1000 * 1000))
        out = {"counts": np.array([len(n), segments, 0, int(pn.max()), int(np.count_nonzero(c)), twins]),
               "line": None}
        if case["pn"]:
            out["pn"] = pn
        return out
    return None
