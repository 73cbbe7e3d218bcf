"""Measured cases: the enumeration jobs that programs give this engine, through its public entry points
(warlib, autotune.cached_tune, serve.Server).

A job is a range of ranks of one space (deals or canonical positions of n cards).  The range of a case has
a fixed length and starts where the seed says, as the spans of a long run, the slices of a sharded run and
the jobs of a server do.  Outputs are the job's exact counts and histograms.
"""
import math
import os
import random
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "endless-games-of-war_b200"))

import autotune  # noqa: E402
import serve  # noqa: E402
import warlib  # noqa: E402

SPAN = (1 << 32) - (1 << 25)     # ranks per engine call of the drop-in programs (war_gpu.py, war17.py)


def listed():
    return [
        # a small job: part of the 10-card table, where the call itself is most of the time
        {"name": "deals10_small", "kind": "deals", "n": 10, "rule": 0, "half": False, "count": 300007},
        # an ordinary slice of 11 cards with the loser's card first (--rule 1), a few million deals
        {"name": "deals11_rule1", "kind": "deals", "n": 11, "rule": 1, "half": False, "count": 5000011},
        # a shard of the 13-card table, 1e8 deals
        {"name": "deals13_shard", "kind": "deals", "n": 13, "rule": 0, "half": False, "count": 100000007},
        # the 13-card table from where an interrupted run left off (the reference's progress is in steps of
        # 256 x 256 deals) to its end: "count" is the most that is left, the seed says how far the run was
        {"name": "deals13_resumed", "kind": "resumed", "n": 13, "rule": 0, "half": False, "count": 6227020800},
        # one span of the 14-card run with --half
        {"name": "deals14_half_span", "kind": "deals", "n": 14, "rule": 0, "half": True, "count": SPAN},
        # one span of the 15-card run
        {"name": "deals15_span", "kind": "deals", "n": 15, "rule": 0, "half": False, "count": SPAN},
        # canonical scans with --distinct --shape: part of the 11-card table, and a long slice of 14 cards
        {"name": "canon11_small", "kind": "canon", "n": 11, "rule": 0, "count": 2000003},
        {"name": "canon14_slice", "kind": "canon", "n": 14, "rule": 0, "count": 3000000019},
        # 17-card deals on the held-out-card engine: the length of the recorded 17-card slices
        {"name": "held17_slice", "kind": "held", "n": 17, "rule": 0, "count": 1000000000},
        # the 5-bit-pile engine: the streak test at 17 cards, Brent with the cycle lengths at 18
        {"name": "wide17_streak", "kind": "wide", "n": 17, "rule": 0, "det": "streak", "count": 200000003},
        {"name": "wide18_brent", "kind": "wide", "n": 18, "rule": 1, "det": "brent", "count": 50000017},
        # a burst of jobs of several sizes on the job server
        {"name": "serve_burst", "kind": "serve", "jobs": 24, "longest": 30000000},
    ]


def draw(rng):
    def count(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(["deals", "deals", "deals", "canon", "canon", "held", "wide", "wide", "serve"])
    if kind == "deals":
        n = rng.choice([9, 10, 11, 12, 13, 14, 15, 16])
        return {"kind": kind, "n": n, "rule": rng.choice([0, 0, 1]), "half": n % 2 == 0 and rng.random() < 0.5,
                "count": count(1e5, min(math.factorial(n) - 1, SPAN))}
    if kind == "canon":
        n = rng.choice([10, 11, 12, 13, 14])
        return {"kind": kind, "n": n, "rule": rng.choice([0, 0, 1]),
                "count": count(1e5, min(math.factorial(n - 1) * (n - 1) - 1, 3000000019))}
    if kind == "held":
        return {"kind": kind, "n": 17, "rule": rng.choice([0, 1]), "count": count(1e5, 1e9)}
    if kind == "wide":
        n = rng.choice([17, 18, 19, 20])
        det = rng.choice(["brent", "floyd"] + (["streak"] if n % 2 else []))
        return {"kind": kind, "n": n, "rule": 0 if det == "streak" else rng.choice([0, 1]), "det": det,
                "count": count(1e5, 1e8)}
    return {"kind": kind, "jobs": rng.randrange(4, 33), "longest": count(1e6, 3e7)}


class Jobs:
    """What a program keeps between calls: the job, its tune, and (serving) the running server."""

    def __init__(self, job=None, tune=None, det=None, jobs=None, server=None):
        self.job, self.tune, self.det, self.jobs, self.server = job, tune, det, jobs, server

    def __del__(self):
        if self.server is not None:
            self.server.close()


def job_of(case, seed):
    rnd = random.Random(seed * 7919 + 17)
    n, kind = case["n"], case["kind"]
    mode = warlib.CANON if kind == "canon" else warlib.DEALS
    total, count = warlib.space_size(n, mode), case["count"]
    if kind == "resumed":
        lo = 65536 * rnd.randrange(0, 4096)
        hi = count
    else:
        lo = rnd.randrange(0, total - count + 1)
        hi = lo + count
    flags = warlib.F_HALF if case.get("half") else 0
    if kind == "canon":
        return warlib.make_job(n, mode, case["rule"], warlib.F_DISTINCT | warlib.F_SHAPE, lo, hi, hbins=256, dbins=4096)
    return warlib.make_job(n, mode, case["rule"], flags, lo, hi, hbins=0 if case.get("det") in ("floyd", "streak") else 256)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        jobs = [j for _, j in serve.poisson_stream(case["jobs"], 1000.0, seed=seed, lmax=case["longest"])]
        return Jobs(jobs=jobs, server=serve.Server(mem_budget=4 << 30))
    job = job_of(case, seed)
    tune = None
    if kind in ("deals", "resumed", "canon"):
        tune = autotune.cached_tune(job.n, job.mode, job.rule, job.flags)
    return Jobs(job, tune, {"brent": warlib.DET_BRENT, "floyd": warlib.DET_FLOYD, "streak": warlib.DET_STREAK}.get(case.get("det")))


def whole(r, names, dist=False):
    """A result's counts and histograms."""
    out = {"counts": np.array([getattr(r, k) for k in names], dtype=np.int64),
           "hist": np.frombuffer(r.hist, dtype=np.int64)[:r.hbins], "endhist": np.frombuffer(r.endhist, dtype=np.int64)}
    if dist:
        out["dhist"] = np.frombuffer(r.dhist, dtype=np.int64)[:r.dbins]
    return out


BASIC = ("cyc", "done", "maxfin")
CANON = BASIC + ("oncycle", "distinct_min", "shape_nonstd", "shape_unchecked")


def run(state):
    if state.server is not None:
        ids = [state.server.submit(j) for j in state.jobs]
        results = [r for r, _ in state.server.wait_all(ids)]
        return {"counts": np.array([[getattr(r, k) for k in CANON] for r in results], dtype=np.int64),
                "hist": np.stack([np.frombuffer(r.hist, dtype=np.int64)[:256] for r in results]),
                "dhist": np.stack([np.frombuffer(r.dhist, dtype=np.int64)[:256] for r in results]),
                "endhist": np.stack([np.frombuffer(r.endhist, dtype=np.int64) for r in results])}
    job = state.job
    if state.det is not None:
        return whole(warlib.enumerate_wide(job, state.det), BASIC + ("undetermined", "turns"))
    if job.n == 17:
        return whole(warlib.enumerate_held(job), BASIC + ("turns",))
    r = warlib.enumerate_job(job, state.tune)
    return whole(r, CANON, True) if job.mode == warlib.CANON else whole(r, BASIC)


# Turns of an average game (Brent, the reference's schedule), by cards; 110.29 at 13 is the recorded total.
TURNS = {9: 38.13, 10: 26.31, 11: 30.46, 12: 20.86, 13: 110.29, 14: 21.0, 15: 110.0, 16: 30.0, 17: 163.5, 18: 40.0,
         19: 160.0, 20: 40.0}
CANON_TURNS = {9: 40.0, 10: 30.0, 11: 35.0, 12: 25.0, 13: 100.0, 14: 35.3, 15: 110.0}


def work(case):
    """Bytes: the job and its result.  Operations: what a path that plays every position does, 22 integer
    operations per turn; a path that decides positions together needs fewer."""
    if case["kind"] == "serve":
        length = (case["longest"] - 1e4) / math.log(case["longest"] / 1e4)
        return {"bytes": case["jobs"] * (64.0 + 8 * (256 * 2 + 1024)), "flops": 22.0 * 40.0 * length * case["jobs"]}
    n, canon = case["n"], case["kind"] == "canon"
    turns = CANON_TURNS[n] if canon else TURNS[n]
    return {"bytes": 64.0 + 8 * (256 + 1024 + (4096 if canon else 0)), "flops": 22.0 * turns * case["count"]}


# ---- the same counts in plain numpy, for jobs small enough ------------------------------------------

def unranked(lo, hi, m):
    """The permutations of 0..m-1 of lexicographic ranks lo..hi-1, one per row."""
    r = np.arange(lo, hi, dtype=np.uint64)
    left = np.tile(np.arange(m, dtype=np.uint8), (hi - lo, 1))
    out = np.empty((hi - lo, m), dtype=np.uint8)
    for i in range(m):
        f = np.uint64(math.factorial(m - 1 - i))
        d = (r // f).astype(np.int64)
        r = r % f
        out[:, i] = left[np.arange(len(left)), d]
        keep = np.arange(m - i)[None, :] != d[:, None]
        left = left[keep].reshape(len(left), m - i - 1)
    return out


def exact(case, seed):
    if case["kind"] not in ("deals", "held") or case["count"] > 400000 or case["n"] > 15:
        return None
    job = job_of(case, seed)
    n, one, four = job.n, np.uint64(1), np.uint64(4)
    p = unranked(job.lo, job.hi, n)
    if job.flags & warlib.F_HALF:
        p = p[np.argmax(p, axis=1) % 2 == 0]
    la, lb = (n + 1) // 2, n // 2
    a = np.full(len(p), 1 << (4 * la), dtype=np.uint64)      # piles: card i in nibble i, a 1 above the last
    b = np.full(len(p), 1 << (4 * lb), dtype=np.uint64)
    for i in range(n):
        c = p[:, i].astype(np.uint64) << np.uint64(4 * (i // 2))
        if i % 2:
            b |= c
        else:
            a |= c
    q = np.full(len(p), la, dtype=np.int64)                  # player 1's cards
    hist, endhist = np.zeros(job.hbins, dtype=np.int64), np.zeros(warlib.WAR_EBINS, dtype=np.int64)
    done, cyc, maxfin, t, saved, mark = len(p), 0, 0, 0, 0, 1
    ta, tb = a.copy(), b.copy()
    while len(a):
        t += 1
        x, y = a & np.uint64(15), b & np.uint64(15)
        w = x > y
        hi, lo = np.maximum(x, y), np.minimum(x, y)
        pair = (lo | (hi << four)) if job.rule else (hi | (lo << four))
        at = np.where(w, q - 1, n - q - 1).astype(np.uint64) * four
        put = ((pair ^ np.uint64(0x101)) << at)
        a = (a >> four) ^ np.where(w, put, np.uint64(0))
        b = (b >> four) ^ np.where(w, np.uint64(0), put)
        q = np.where(w, q + 1, q - 1)
        end = (q == 0) | (q == n)
        again = (a == ta) & (b == tb) & ~end
        if end.any():
            maxfin = t
            endhist[min(t, warlib.WAR_EBINS - 1)] += int(end.sum())
        if again.any():
            cyc += int(again.sum())
            hist[min(t - saved, job.hbins - 1)] += int(again.sum())
        go = ~(end | again)
        if not go.all():
            a, b, q, ta, tb = a[go], b[go], q[go], ta[go], tb[go]
        if t == mark:
            ta, tb, saved, mark = a.copy(), b.copy(), t, 2 * mark + 1
    return {"counts": np.array([cyc, done, maxfin], dtype=np.int64), "hist": hist, "endhist": endhist}
