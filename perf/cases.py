"""Performance cases of the Goldbach verifier, through its public entry points.

Each case is one call (or one burst of serving requests) as a program that
uses the library makes it: the Python view of the C-ABI where it returns
arrays, the C-ABI itself where the caller owns the buffers.  Kinds:

  single   gb_check_single_batch: minimal (p, q) of a batch of even n
  range    gb_verify_range: every even n of [start, limit]
  windows  gb_verify_windows: many independent ranges in one batch
  counts   gb_goldbach_counts: partition counts c(n)
  big      gb_check_big: one even n beyond 2^64
  serve    gb_submit / gb_wait: a burst of mixed requests to a running server

The programs keep one context (its resident prime tables) and, for serving,
one running server; the inputs of every state are drawn from its seed.
All outputs are whole numbers.
"""
import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

U64_TOP = 2**64 - 2


def _package():
    mod = sys.modules.get("goldbach_gpu_b200")
    if mod is None:
        spec = importlib.util.spec_from_file_location(
            "goldbach_gpu_b200", os.path.join(_ROOT, "goldbach-gpu_b200", "__init__.py"))
        mod = importlib.util.module_from_spec(spec)
        sys.modules["goldbach_gpu_b200"] = mod
        spec.loader.exec_module(mod)
    return mod


_handles = {}


def _context():
    """The context such a program keeps, with the tables for n up to 1e18."""
    if "context" not in _handles:
        _handles["context"] = _package().Context(0, max_n=10**18)
    return _handles["context"]


def _server():
    """A running server over a context of its own (n up to 2^64 - 2), its lanes
    polling 20 ms before they block, as the serving benchmark runs it."""
    if "server" not in _handles:
        ctx = _package().Context(0, max_n=U64_TOP)
        ctx.serve_start(max_n=U64_TOP, spin_us=20000, pool_bytes=4 << 30)
        _handles["server"] = ctx
    return _handles["server"]


# -- the cases ---------------------------------------------------------------

def listed():
    return [
        # one query of a command line or an interactive caller (single_check <n>):
        # latency is all that counts
        {"name": "single_1", "kind": "single", "count": 1, "bits": 64, "on_device": False},
        # a service's ordinary batch, odd-sized, host arrays in and out
        {"name": "single_3001", "kind": "single", "count": 3001, "bits": 64, "on_device": False},
        # a million queries uniform in [4, 2^64 - 2], resident on the device
        {"name": "single_1e6", "kind": "single", "count": 1_000_000, "bits": 64, "on_device": True},
        # one reported segment (the default 1e7 even n) below 1e12, summary, histogram
        # and per-segment figures on the host: a resumed run's smallest unit
        {"name": "range_segment", "kind": "range", "top": 10**12, "count": 10_000_000, "seg_size": 10_000_000,
         "per_n": False},
        # every even n in [4, 1e9] with the minimal p of each and the verified bitmap, seg-size 2^26
        {"name": "range_1e9_per_n", "kind": "range", "top": 10**9, "count": 499_999_999, "seg_size": 1 << 26,
         "per_n": True},
        # every even n in [4, 1e12], seg-size 2^27: the headline run
        {"name": "range_1e12", "kind": "range", "top": 10**12, "count": 499_999_999_999, "seg_size": 1 << 27,
         "per_n": False},
        # a slice far out, beyond what has been verified so far in one go (--start=A), ragged
        {"name": "range_far", "kind": "range", "top": 10**15, "count": 40_000_003, "seg_size": 10_000_000,
         "per_n": False},
        # 4096 windows at offsets uniform in [1e15, 1e18], widths log-uniform in [2^10, 2^24]
        {"name": "windows_4096", "kind": "windows", "windows": 4096, "lo": 10**15, "hi": 10**18, "wlo": 10.0,
         "whi": 24.0, "per_n": False},
        # a small batch with the minimal p of every n returned
        {"name": "windows_61_per_n", "kind": "windows", "windows": 61, "lo": 10**15, "hi": 10**18, "wlo": 10.0,
         "whi": 18.0, "per_n": True},
        # partition counts of 4096 consecutive even n near 1e9
        {"name": "counts_4096", "kind": "counts", "top": 10**9, "count": 4096},
        # one even n of 512 bits (big_check)
        {"name": "big_512", "kind": "big", "bits": 512},
        # a burst of mixed requests, 70% single n up to 2^64 and 30% ranges of 2^8 to
        # 2^22 even n at offsets up to 1e19, to a running server
        {"name": "serve_512", "kind": "serve", "requests": 512, "whi": 22.0},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "single", "range", "range", "range", "windows", "windows", "counts", "big", "serve"])
    if kind == "single":
        return {"kind": kind, "count": _log_uniform(rng, 1, 1_000_000), "bits": rng.randint(36, 64),
                "on_device": rng.random() < 0.4}
    if kind == "range":
        top = _log_uniform(rng, 10**8, 10**17)
        per_n = rng.random() < 0.3
        most = 1 << 26 if top > 10**13 or per_n else 1 << 34
        count = min(_log_uniform(rng, 1 << 14, most), top // 2 - 1001)
        return {"kind": kind, "top": top, "count": count, "seg_size": _log_uniform(rng, 10**6, 10**8), "per_n": per_n}
    if kind == "windows":
        per_n = rng.random() < 0.4
        return {"kind": kind, "windows": _log_uniform(rng, 1, 256 if per_n else 4096), "lo": 10**12,
                "hi": _log_uniform(rng, 10**13, 10**18), "wlo": 8.0,
                "whi": round(rng.uniform(10.0, 18.0 if per_n else 24.0), 2), "per_n": per_n}
    if kind == "counts":
        return {"kind": kind, "top": _log_uniform(rng, 10**6, 2 * 10**9), "count": _log_uniform(rng, 32, 4096)}
    if kind == "big":
        return {"kind": kind, "bits": rng.randint(80, 512)}
    return {"kind": kind, "requests": _log_uniform(rng, 8, 1024), "whi": round(rng.uniform(10.0, 22.0), 2)}


# -- inputs ------------------------------------------------------------------

def _even_below(rng, bits, count):
    """count even n, uniform in [4, 2^bits - 2]."""
    return rng.integers(2, 2 ** (bits - 1), size=count, dtype=np.uint64) * np.uint64(2)


def _range_bounds(case, seed):
    """The case's range, moved down by a little that the seed gives (its count is
    the same for every seed; a range from the bottom starts at 4 or just above)."""
    shift = int(np.random.default_rng(seed).integers(0, 1000))
    top = case["top"] - case["top"] % 2
    count = min(case["count"], top // 2 - 1001)
    limit = top - 2 * shift
    return limit - 2 * (count - 1), limit


def _windows_input(case, seed):
    """Offsets by the seed, widths by the case (the outputs' sizes do not hang on the seed)."""
    n = case["windows"]
    starts = np.random.default_rng(seed).integers(case["lo"] // 2, case["hi"] // 2, size=n,
                                                  dtype=np.uint64) * np.uint64(2)
    widths = np.random.default_rng([n, int(case["whi"] * 100)])
    counts = np.exp2(widths.uniform(case["wlo"], case["whi"], size=n)).astype(np.uint64)
    return starts, counts


def _counts_start(case, seed):
    shift = int(np.random.default_rng(seed).integers(0, 1000))
    return max(4, case["top"] - case["top"] % 2 - 2 * (case["count"] + shift))


def _big_n(case, seed):
    rng = np.random.default_rng(seed)
    words = [int(x) for x in rng.integers(0, 2**32, size=(case["bits"] + 31) // 32, dtype=np.uint64)]
    n = sum(w << (32 * i) for i, w in enumerate(words)) & ((1 << case["bits"]) - 1)
    return (n | (1 << (case["bits"] - 1))) & ~1


def _requests(case, seed):
    rng = np.random.default_rng(seed)
    m = case["requests"]
    single = rng.random(m) < 0.7
    a = np.where(single, rng.integers(2, 2**63, size=m, dtype=np.uint64),
                 rng.integers(2, 5 * 10**18, size=m, dtype=np.uint64)) * np.uint64(2)
    counts = np.where(single, 1, np.exp2(rng.uniform(8.0, case["whi"], size=m))).astype(np.uint64)
    return single, a, counts


def prepare(case, seed):
    gb = _package()
    kind = case["kind"]
    state = {"case": case, "gb": gb}
    if kind == "single":
        state["ctx"] = _context()
        n = _even_below(np.random.default_rng(seed), case["bits"], case["count"])
        state["n"] = n
        if case["on_device"]:
            state["n"] = torch.from_numpy(n.view(np.int64)).cuda()
            state["p"] = torch.zeros(case["count"], dtype=torch.int64, device="cuda")
            state["q"] = torch.zeros(case["count"], dtype=torch.int64, device="cuda")
    elif kind == "range":
        state["ctx"] = _context()
        start, limit = _range_bounds(case, seed)
        state["start"], state["limit"] = start, limit
        if case["per_n"]:  # the caller's device buffers
            count = (limit - start) // 2 + 1
            segs = -(-count // case["seg_size"])
            state["out"] = {
                "min_p": torch.zeros(count, dtype=torch.int32, device="cuda"),
                "verified_bits": torch.zeros(-(-count // 32), dtype=torch.int32, device="cuda"),
                "minp_hist": torch.zeros(gb.GB_HIST_BINS, dtype=torch.int64, device="cuda"),
                "seg_fallbacks": torch.zeros(segs, dtype=torch.int32, device="cuda"),
                "seg_failures": torch.zeros(segs, dtype=torch.int32, device="cuda"),
            }
    elif kind == "windows":
        state["ctx"] = _context()
        starts, counts = _windows_input(case, seed)
        n = len(starts)
        w = np.zeros((n, 2), np.uint64)
        w[:, 0], w[:, 1] = starts, counts
        state["w"] = w
        state["results"] = np.zeros((n, 4), np.uint64)
        state["min_p"] = np.zeros(int(counts.sum()), np.uint32) if case["per_n"] else None
    elif kind == "counts":
        state["ctx"] = _context()
        state["start"] = _counts_start(case, seed)
    elif kind == "big":
        state["ctx"] = _context()
        state["n"] = _big_n(case, seed)
    else:
        state["ctx"] = _server()
        single, a, counts = _requests(case, seed)
        state["kinds"] = np.where(single, gb.GB_REQ_SINGLE, gb.GB_REQ_RANGE).astype(np.int32)
        state["a"], state["counts"] = a, counts
        state["responses"] = (gb.Response * len(a))()
    return state


# -- one pass ----------------------------------------------------------------

def run(state):
    case, gb, ctx = state["case"], state["gb"], state["ctx"]
    kind = case["kind"]
    if kind == "single":
        if case["on_device"]:
            _, _, r = ctx.check_single(None, device_ptrs=(state["n"], state["p"], state["q"]))
            return {"p": state["p"], "q": state["q"], "found": r.found, "max_p": r.max_p}
        p, q, r = ctx.check_single(state["n"])
        return {"p": p.view(np.int64), "q": q.view(np.int64), "found": r.found, "max_p": r.max_p}
    if kind == "range":
        if case["per_n"]:
            got = ctx.verify_range(state["start"], state["limit"], seg_size=case["seg_size"], p_small=10**8,
                                   device_out=state["out"])
            arrays = dict(state["out"])
        else:
            got = ctx.verify_range(state["start"], state["limit"], seg_size=case["seg_size"], want_seg=True)
            arrays = {"minp_hist": got.hist.view(np.int64), "seg_fallbacks": got.seg_fallbacks.view(np.int32),
                      "seg_failures": got.seg_failures.view(np.int32)}
        figures = ("checked", "verified", "phase2_fallbacks", "failures", "first_failure_n", "max_minp",
                   "num_segments")
        return arrays | {f: got.result[f] for f in figures}
    if kind == "windows":
        w, results, min_p = state["w"], state["results"], state["min_p"]
        opts, summary = gb.WindowsOpts(), gb.WindowsSummary()
        st = ctx.L.gb_verify_windows(
            ctx._h, ctypes.cast(w.ctypes.data, ctypes.POINTER(gb.Window)), len(w), ctypes.byref(opts),
            ctypes.cast(results.ctypes.data, ctypes.POINTER(gb.WindowResult)),
            None if min_p is None else min_p.ctypes.data, ctypes.byref(summary))
        if st != gb.GB_OK:
            raise gb.GbError(st, ctx.L.gb_last_error(ctx._h).decode())
        out = {"results": results.view(np.int64), "total_n": summary.total_n, "failures": summary.failures}
        return out if min_p is None else out | {"min_p": min_p.view(np.int32)}
    if kind == "counts":
        return ctx.goldbach_counts(state["start"], case["count"]).view(np.int64)
    if kind == "big":
        p, q, _ = ctx.check_big(state["n"])
        return {"p": p, "q": _limbs(q, case["bits"])}
    responses = state["responses"]
    tickets = ctx.submit(state["kinds"], state["a"], state["counts"])
    for i, t in enumerate(tickets.tolist()):
        st = ctx.L.gb_wait(ctx._h, t, ctypes.byref(responses[i]), 60000)
        if st != gb.GB_OK:
            raise gb.GbError(st, "request %d" % i)
    got = np.frombuffer(responses, dtype=[("status", "<i4"), ("kind", "<i4"), ("figures", "<i8", (6,)),
                                          ("latency_us", "<f8"), ("lane", "<u4"), ("batch", "<u4")])
    return {"status": got["status"], "figures": got["figures"]}


def _limbs(v, bits):
    return np.array([(v >> (32 * i)) & 0xFFFFFFFF for i in range((bits + 31) // 32)], dtype=np.int64)


# -- the work of a pass ------------------------------------------------------
# Bytes: inputs and outputs.  Flops: 32-bit integer operations, by what each
# path cannot do without (no floating-point operation occurs anywhere).

_PRODUCT = 20  # 32-bit multiply-adds of one 64-bit Montgomery product


def _single_ops(n_count, bits):
    # ~ ln(n) / 2 candidates, of which a sieve leaves about an eighth of ln(n); a
    # strong test is `bits` squarings, and the one that is prime takes three times that
    return n_count * (0.12 * bits * 0.69 + 3) * bits * _PRODUCT


def _range_ops(count, top):
    # a word test of five operations for every 32 (n, p) pairs tried, one mark for
    # every prime factor of a window number, one offset per sieving prime and 2^20 n
    tries = 0.6 * math.log(top)
    marks = 2 * math.log(max(2.0, math.log(top) / 2))
    root = math.sqrt(top)
    return count * (tries * 5 / 32 + marks) + 8 * root / math.log(root) * math.ceil(count / 2**20)


def work(case):
    kind = case["kind"]
    if kind == "single":
        return {"bytes": 24 * case["count"], "flops": _single_ops(case["count"], case["bits"])}
    if kind == "range":
        count = min(case["count"], case["top"] // 2 - 1001)
        out = count * 4.125 if case["per_n"] else 0
        return {"bytes": 4096 * 8 + 8 * -(-count // case["seg_size"]) + out, "flops": _range_ops(count, case["top"])}
    if kind == "windows":
        wlo, whi = 2.0 ** case["wlo"], 2.0 ** case["whi"]
        mean = (whi - wlo) / math.log(whi / wlo)
        total = mean * case["windows"]
        out = total * 4 if case["per_n"] else 0
        # a window is sieved in full, or sieved a little and its primes tested
        root = math.sqrt(case["hi"])
        per_window = min(8 * root / math.log(root), 2 * mean / math.log(case["hi"]) * 200 * _PRODUCT)
        return {"bytes": 48 * case["windows"] + out,
                "flops": _range_ops(total, 10**12) + case["windows"] * per_window}
    if kind == "counts":
        # 32 pairs (p, n - p), both odd and coprime to 3, to a word operation of four
        return {"bytes": case["top"] / 16 + 8 * case["count"], "flops": case["count"] * case["top"] / 9 * 4 / 32}
    if kind == "big":
        limbs = case["bits"] / 32
        return {"bytes": 12 * limbs, "flops": (0.06 * case["bits"] + 12) * case["bits"] * 4 * limbs * limbs}
    mean = (2.0 ** case["whi"] - 2.0**8) / math.log(2.0 ** (case["whi"] - 8))
    m = case["requests"]
    return {"bytes": m * 96, "flops": _single_ops(0.7 * m, 64) + 0.3 * m * mean * 2 / 43 * 200 * _PRODUCT}


# -- what the outputs are, in plain Python and numpy --------------------------

def _primes(limit):
    s = np.ones(limit + 1, bool)
    s[:2] = False
    for p in range(2, math.isqrt(limit) + 1):
        if s[p]:
            s[p * p::p] = False
    return np.flatnonzero(s)


_BASES = (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37)


def _is_prime(q):
    if q < 2:
        return False
    for b in _BASES:
        if q % b == 0:
            return q == b
    d, s = q - 1, 0
    while d % 2 == 0:
        d, s = d // 2, s + 1
    for b in _BASES:
        x = pow(b, d, q)
        if x in (1, q - 1):
            continue
        for _ in range(s - 1):
            x = x * x % q
            if x == q - 1:
                break
        else:
            return False
    return True


def _minimal_p(n, primes):
    if n == 4:
        return 2
    for p in primes:
        if p > n // 2:
            return 0
        if p > 2 and _is_prime(n - p):
            return p
    return 0


def _exact_range(case, seed):
    start, limit = _range_bounds(case, seed)
    count = (limit - start) // 2 + 1
    halo = 1 << 15
    lo = max(3, start - halo) | 1
    odd = np.ones((limit - lo) // 2 + 1, bool)  # bit i <-> lo + 2i
    for p in _primes(math.isqrt(limit))[1:].tolist():
        m = max(p * p, -(-lo // p) * p)
        odd[(m + p * (m % 2 == 0) - lo) // 2::p] = False
    primes = _primes(halo)
    min_p = np.zeros(count, np.int64)
    left = np.arange(count)
    if start == 4:
        min_p[0], left = 2, left[1:]
    for p in primes[1:].tolist():
        n = start + 2 * left
        at = (n - p - lo) // 2
        hit = (2 * p <= n) & (at >= 0) & odd[np.maximum(at, 0)]
        min_p[left[hit]] = p
        left = left[~hit]
        if not len(left):
            break
    if len(left):
        return None
    segs = -(-count // case["seg_size"])
    hist = np.zeros(4096, np.int64)
    np.add.at(hist, np.searchsorted(primes, min_p), 1)
    got = {"minp_hist": hist, "seg_fallbacks": np.zeros(segs, np.int32), "seg_failures": np.zeros(segs, np.int32),
           "checked": count, "verified": count, "phase2_fallbacks": 0, "failures": 0, "first_failure_n": 0,
           "max_minp": int(min_p.max()), "num_segments": segs}
    if case["per_n"]:
        bits = np.zeros(-(-count // 32) * 32, np.uint8)
        bits[:count] = 1
        got["min_p"] = min_p.astype(np.int32)
        got["verified_bits"] = np.packbits(bits, bitorder="little").view(np.int32)
    return got


def exact(case, seed):
    kind = case["kind"]
    if kind == "single" and case["count"] <= 4096:
        n = _even_below(np.random.default_rng(seed), case["bits"], case["count"])
        primes = _primes(1 << 14).tolist()
        p = np.array([_minimal_p(int(x), primes) for x in n], np.uint64)
        return {"p": p.view(np.int64), "q": (n - p).view(np.int64), "found": int((p > 0).sum()), "max_p": int(p.max())}
    if kind == "range" and case["count"] <= 10_000_000 and case["top"] <= 2 * 10**12:
        return _exact_range(case, seed)
    if kind == "big":
        n = _big_n(case, seed)
        p = _minimal_p(n, _primes(1 << 18).tolist())
        return {"p": p, "q": _limbs(n - p, case["bits"])} if p else None
    return None
