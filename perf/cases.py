"""Performance cases of the census framework: what its users have it compute,
through its public entry points, from single calls to whole blocks.

A case is a dict of plain values.  `op` names the entry point:

  census    Census.raw      consecutive primes through the filter or, for small
                            primes, the dense scan (mode "auto"), or through the
                            dense scan only (mode "dense", the audits' re-run)
  worker    Census.profiles the line-protocol worker's batch: certified records
                            as Python objects, no A4
  uneven    Census.raw      many short windows, starts log-uniform over a range,
                            in one call
  interval  Census.interval every prime of [lo, hi): device sieve + census
  a4        Census.a4       the A4 worker's batch
  wide      Census64.raw    primes above 2^32
  serve     serving.Server  a burst of requests submitted together, all fetched

`lo` and `span` give the range in which the seed places the window's start,
`count` the primes (for `uneven` those of one window, for `serve` those of the
largest request).  Profiles come back as one row of 8 orders (2..9, zeros where
r does not divide p - 1) per prime.
"""
from __future__ import annotations

import math
import random

import numpy as np

from rabung_atlas32_b200 import sieve
from rabung_atlas32_b200.census import Census, Census64
from rabung_atlas32_b200.serving import Server

TOP = 2 ** 32


def listed():
    return [
        # one prime per call, the per-prime form of the census worker and of the
        # C ABI's baseline_profile: latency and launches
        {"name": "one_prime", "op": "census", "lo": 3_000_000_000, "span": 200_000_000, "count": 1, "mode": "auto",
         "a4": True},
        # small primes: the first blocks of an atlas, the dense scan, a call of
        # a few hundred microseconds
        {"name": "small_primes_256", "op": "census", "lo": 2, "span": 1200, "count": 256, "mode": "auto", "a4": True},
        # the census worker's batch of 128 primes in the upper half of the domain
        {"name": "worker_128", "op": "worker", "lo": 4_200_000_000, "span": 60_000_000, "count": 128},
        # an odd, short request in the middle of the domain
        {"name": "mid_37", "op": "census", "lo": 700_000_000, "span": 40_000_000, "count": 37, "mode": "auto",
         "a4": True},
        # a block of 4096 primes near 2^24
        {"name": "block_2p24", "op": "census", "lo": 16_777_216, "span": 1_000_000, "count": 4096, "mode": "auto",
         "a4": True},
        # a block of 4096 primes just below 2^32: the headline workload
        {"name": "block_top", "op": "census", "lo": 4_290_000_000, "span": 4_800_000, "count": 4096, "mode": "auto",
         "a4": True},
        # the dense scan as the filter's judge: a block's sample re-run near 2^24
        {"name": "dense_2p24_700", "op": "census", "lo": 16_777_216, "span": 1_000_000, "count": 700, "mode": "dense",
         "a4": False},
        # short windows from all over the domain in one call
        {"name": "uneven_40x61", "op": "uneven", "lo": 1 << 16, "span": TOP - (1 << 16), "count": 61, "windows": 40},
        # the supervisor's step: every prime of an interval, device sieve and census
        {"name": "interval_2p28", "op": "interval", "lo": 268_435_456, "span": 4_000_000, "count": 991},
        # the A4 worker's largest batch
        {"name": "a4_4096", "op": "a4", "lo": 4_000_000_000, "span": 200_000_000, "count": 4096},
        # primes above 2^32 (64-bit words)
        {"name": "wide_96", "op": "wide", "lo": 5_300_000_000, "span": 200_000_000, "count": 96, "a4": True},
        # serving: a burst of 24 requests of 1 to 256 primes, starts log-uniform
        # over the domain, sizes in geometric steps
        {"name": "serve_24", "op": "serve", "lo": 1 << 12, "span": TOP - (1 << 12), "count": 256, "requests": 24},
    ]


def _log_int(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    """One more case of the same ranges: the entry point by its share of use,
    sizes spread over their logarithm."""
    op = rng.choice(["census", "census", "census", "worker", "dense", "uneven", "interval", "a4", "wide", "serve"])
    if op == "worker":
        return {"op": "worker", "lo": _log_int(rng, 1 << 14, 4_200_000_000), "span": 1_000_000,
                "count": _log_int(rng, 1, 128)}
    if op == "census":
        lo = _log_int(rng, 1 << 13, 4_200_000_000)
        return {"op": "census", "lo": lo, "span": max(1000, lo // 64), "count": _log_int(rng, 1, 4096), "mode": "auto",
                "a4": rng.random() < 0.7}
    if op == "dense":                          # at most about a fifth of a second of powers
        lo = _log_int(rng, 1 << 14, 1 << 27)
        return {"op": "census", "lo": lo, "span": max(1000, lo // 64),
                "count": _log_int(rng, 1, max(2, min(2048, (700 << 24) // lo))), "mode": "dense", "a4": False}
    if op == "uneven":
        return {"op": "uneven", "lo": 1 << 16, "span": TOP - (1 << 16), "count": _log_int(rng, 8, 96),
                "windows": rng.randint(5, 48)}
    if op == "interval":
        lo = _log_int(rng, 1 << 13, 4_200_000_000)
        return {"op": "interval", "lo": lo, "span": max(1000, lo // 64), "count": _log_int(rng, 20, 4096)}
    if op == "a4":
        lo = _log_int(rng, 1 << 11, 4_200_000_000)
        return {"op": "a4", "lo": lo, "span": max(1000, lo // 64), "count": _log_int(rng, 1, 4096)}
    if op == "wide":
        return {"op": "wide", "lo": _log_int(rng, TOP + 1, 8_400_000_000), "span": 100_000_000,
                "count": _log_int(rng, 1, 256), "a4": rng.random() < 0.5}
    return {"op": "serve", "lo": 1 << 12, "span": TOP - (1 << 12), "count": _log_int(rng, 8, 512),
            "requests": rng.randint(2, 32)}


# ---------------------------------------------------------------- inputs ----

def _wide_primes(start, count):
    """The first `count` primes >= start (start above 2^32)."""
    out, lo, width = [], start, 1 << 16
    while len(out) < count:
        mark = np.ones(width, dtype=bool)
        for q in sieve.primes_in(2, math.isqrt(lo + width) + 1):
            mark[(-lo) % q::q] = False
        out += [int(x) + lo for x in np.nonzero(mark)[0]]
        lo += width
    return out[:count]


def _window(case, seed):
    rng = random.Random(1_000_003 * seed + 17)
    start = case["lo"] + rng.randrange(max(1, case["span"]))
    if case["op"] == "wide":
        return _wide_primes(start, case["count"])
    return sieve.primes_from(min(start, TOP - 200_000), case["count"])


class _Burst:
    """A serving runtime and a burst of requests; closed with its state."""

    def __init__(self, requests):
        self.server = Server(slots=1, slot_budget_mb=12 * 1024)
        self.requests = requests

    def __del__(self):
        self.server.close()


def prepare(case, seed):
    op = case["op"]
    if op == "serve":
        rng = random.Random(1_000_003 * seed + 29)
        top = case["lo"] + case["span"]
        n = case["requests"]
        reqs = [(min(_log_int(rng, case["lo"], top), TOP - 200_000), int(case["count"] ** (k / max(1, n - 1))))
                for k in range(n)]
        rng.shuffle(reqs)
        return {"case": case, "burst": _Burst(reqs)}
    if op == "uneven":
        rng = random.Random(1_000_003 * seed + 31)
        # starts log-uniform, one per equal slice of the range, so that the
        # windows of any seed cover the domain alike
        a, b, n = math.log(case["lo"]), math.log(case["lo"] + case["span"]), case["windows"]
        starts = [int(math.exp(a + (b - a) * (k + rng.random()) / n)) for k in range(n)]
        ps = [p for s in starts for p in sieve.primes_from(min(s, TOP - 200_000), case["count"])]
        return {"case": case, "engine": Census(), "primes": ps}
    if op == "interval":
        rng = random.Random(1_000_003 * seed + 37)
        lo = case["lo"] + rng.randrange(max(1, case["span"]))
        return {"case": case, "engine": Census(), "lo": lo, "hi": sieve.primes_from(lo, case["count"])[-1] + 1}
    return {"case": case, "engine": Census64() if op == "wide" else Census(), "primes": _window(case, seed)}


# ------------------------------------------------------------------ passes ----

def _by_order(p, rows):
    """One row per prime of p and order 2..9 from the records' rows (in prime
    order, ascending admissible r); zeros where r does not divide p - 1."""
    p = np.asarray(p, dtype=np.int64)
    adm = ((p[:, None] - 1) % np.arange(2, 10) == 0) & (p[:, None] > 2)
    out = np.zeros(adm.shape + rows.shape[1:], dtype=np.int64)
    out[adm] = rows
    return out


def _profiles(recs):
    """(p, r, M, L, witness, K) of codec.Record objects by order, and A4."""
    rows = [(rec.p, v.r, v.M, v.L, v.witness, v.K) for rec in recs for v in rec.profiles]
    ps = [rec.p for rec in recs]
    return (_by_order(ps, np.array(rows, dtype=np.int64).reshape(-1, 6)),
            np.array([rec.a4 for rec in recs], dtype=np.int64))


def run(state):
    case, op = state["case"], state["case"]["op"]
    if op == "serve":
        srv, reqs = state["burst"].server, state["burst"].requests
        ids = {srv.submit(lo, n): k for k, (lo, n) in enumerate(reqs)}
        got = [None] * len(reqs)
        while ids:
            rid = srv.next_done(60_000)
            k = ids.pop(rid)
            got[k] = srv.fetch(rid, reqs[k][1])
        rows, a4 = _profiles([rec for _, recs in got for rec in recs])
        return {"profiles": rows, "a4": a4}
    eng = state["engine"]
    if op == "interval":
        primes, recs = eng.interval(state["lo"], state["hi"])
        rows, a4 = _profiles(recs)
        return {"primes": np.array(primes, dtype=np.int64), "profiles": rows, "a4": a4}
    if op == "a4":
        return np.array(eng.a4(state["primes"]), dtype=np.int64)
    if op == "worker":
        rows, _ = _profiles(eng.profiles(state["primes"], mode="auto", a4=False, verify=True))
        return rows
    # the library's records as 32-bit words
    out, a4, stats = eng.raw(state["primes"], mode=case.get("mode", "auto"), a4=case.get("a4", True))
    recs = np.frombuffer(out, dtype=np.uint32).reshape(len(out), -1)[:stats["n_profiles"]]
    recs = _by_order(state["primes"], recs)
    return {"records": recs, "a4": np.array(a4, dtype=np.int64)} if a4 is not None else {"records": recs}


# -------------------------------------------------------------------- work ----

def work(case):
    """Bytes: the primes read and the records written.  Operations: for a prime
    through the filter, one 32-bit plane test for each 32 positions of the half
    interval and each of its about 3.3 profiles; for the dense scan, a power
    (about 1.4 log2 p products of four multiplies) for each position; for A4,
    the baby and giant steps of the point count (4 p^(1/4) curve operations of
    about 60 products)."""
    op, n = case["op"], case["count"]
    mid = case["lo"] + case["span"] / 2
    if op in ("uneven", "serve"):
        hi = case["lo"] + case["span"]
        mean_p = (hi - case["lo"]) / math.log(hi / case["lo"])
        n = n * case["windows"] if op == "uneven" else max(1, int(case["requests"] * n / math.log(max(3, n))))
    else:
        mean_p = mid
    lg = math.log2(max(4.0, mean_p))
    power = 1.4 * lg * 4
    ops = 0.0
    if op != "a4":
        if case.get("mode") == "dense" or mean_p < 1 << 14:
            ops += n * mean_p / 2 * power
        else:
            ops += n * 3.3 * mean_p / 2 / 32
    if op == "a4" or case.get("a4", op not in ("worker",)):
        ops += n * 4 * mean_p ** 0.25 * 60 * 4
    return {"bytes": float(n * (4 + 4 + (0 if op == "a4" else 3.3 * 32))), "flops": float(ops)}


# ------------------------------------------------------------------- exact ----

def _exact_prime(p):
    """(r, M, L, witness, K) rows and A4 of a small odd prime, from the index
    table of a primitive root."""
    fac = [q for q in range(2, p) if (p - 1) % q == 0 and all(q % d for d in range(2, math.isqrt(q) + 1))]
    g = next(a for a in range(1, p) if all(pow(a, (p - 1) // q, p) != 1 for q in fac) or p == 3 and a == 2)
    ind = np.zeros(p, dtype=np.int64)
    x = 1
    for k in range(p - 1):
        ind[x] = k
        x = x * g % p
    rows = []
    for r in range(2, 10):
        if (p - 1) % r:
            continue
        c = ind[1:] % r
        edges = np.concatenate([[0], np.nonzero(np.diff(c))[0] + 1, [p - 1]])
        lens = np.diff(edges)
        M = int(lens.max())
        w = min(min(int(s) + 1, p - (int(s) + M)) for s in edges[:-1][lens == M])
        L = int(lens[0])
        K = max(M + 1, 2 * L + 2 if ((p - 1) // 2) % r == 0 else L + 2)
        rows.append((r, M, L, w, K))
    q = ind[1:] % 2
    a4 = int(np.sum((q[:-3] == q[1:-2]) & (q[1:-2] == q[2:-1]) & (q[2:-1] == q[3:]))) if p > 4 else 0
    return rows, a4


def exact(case, seed):
    if case["op"] != "census" or not case.get("a4") or (case["lo"] + case["span"]) * case["count"] > 2_000_000:
        return None
    primes = _window(case, seed)
    recs, a4 = [], []
    for p in primes:
        rows, a = _exact_prime(p) if p > 2 else ([], 0)
        recs += [(p, r, M, L, w, 0, K & 0xFFFFFFFF, K >> 32) for r, M, L, w, K in rows]
        a4.append(a)
    recs = np.array(recs, dtype=np.int64).reshape(-1, 8)
    return {"records": _by_order(primes, recs), "a4": np.array(a4, dtype=np.int64)}
