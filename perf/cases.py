"""Workloads of the sieve for timing: what users have it do, through the package's public entry points.

The sizes are this repository's own: the three benchmark searches, the setup-bound searches and the batch
of uneven searches of bench.py, and the reference's self-test ranges.  A case's kind names the entry point:

  search    pfc.sieve() on the user's context: tables, candidates, setup, walk, hits, verification, checksum
  segments  the reference's host loop: one job kept, its p range walked segment by segment, hits drained
            and finalized after each
  batch     many uneven searches through one pfc.Batch, then every search's totals and hits
  verify    pfc.verify_factors(): the device re-verification of a finished search's hits

Modes are the reference's: 1 for n!, 2 for n#, 4 for n!/n#, 5 for n! and n!/n# together.  The seed moves
the p range (a sieve's user sweeps p at a fixed n range), and for a batch draws the searches.
"""
import math
import os
import random

import numpy as np

import pfcsieve_gb300 as pfc
from pfcsieve_gb300 import serving

SPLIT32 = 2**31      # candidates below take 32-bit arithmetic
LAZY_END = 2**64 // 3   # and at or above this the canonical 64-bit one


def listed():
    return [
        # the smallest calls: a short search a user runs to see that everything works, all latency
        _search("search-tiny", 1, 101, 2000, 10**6, 10**6 + 50000),
        # the benchmark's small search, 1.2e9 pairs
        _search("search-factorial-1e7", 1, 101, 20000, 10**7, 11 * 10**6),
        # the headline search: 9.6e11 pairs of the combined walk
        _search("search-combined-1e9", 5, 101, 200000, 10**9, 10**9 + 10**8),
        # the benchmark's n# search with candidates near 2^62
        _search("search-primorial-2e62", 2, 101, 10**6, 2**62, 2**62 + 5 * 10**7),
        # n!/n# at the p and n of the self-test's compositorial ranges (p near 10^12, n from 700,000)
        _search("search-compositorial-1e12", 4, 700000, 900000, 10**12, 10**12 + 2 * 10**7),
        # deep factorial sieving: large start n and a moderate n range, so setup and walk both count
        _search("search-factorial-1e13", 1, 10**6, 1050000, 10**13, 10**13 + 10**7),
        # short n ranges from a large n0, where the start residues are the work (32- and 64-bit p)
        _search("search-setup-1e9", 5, 5 * 10**6, 5001000, 10**9, 10**9 + 4 * 10**6),
        _search("search-setup-2e40", 1, 9 * 10**6, 9001000, 2**40, 2**40 + 4 * 10**6),
        # the top of the p range, above 2^64/3
        _search("search-factorial-top", 1, 101, 20000, 15 * 10**18, 15 * 10**18 + 4 * 10**6),
        # the command line's loop on the self-test's combined range near 10^11 (an odd n length)
        {"name": "segments-combined-1e11", "kind": "segments", "mode": 5, "nmin": 96000, "nmax": 136777,
         "pmin": 10**11, "pmax": 10**11 + 8 * 10**6, "parts": 4},
        # a queue of uneven searches served together, the batch workload's mix at smaller lengths
        {"name": "batch-mixed-24", "kind": "batch", "count": 24, "n0": 10**7, "nlen": 10**5, "plen": 10**7},
        # device check of about ten thousand factors
        {"name": "verify-combined-1e6", "kind": "verify", "mode": 5, "nmin": 101, "nmax": 200000,
         "pmin": 10**6, "pmax": 1200000},
    ]


def _search(name, mode, nmin, nmax, pmin, pmax):
    return {"name": name, "kind": "search", "mode": mode, "nmin": nmin, "nmax": nmax, "pmin": pmin, "pmax": pmax,
            "verify": "device" if nmax > 10**6 else "cpu"}


def _candidates(case):
    return (case["pmax"] - case["pmin"]) / math.log(case["pmin"]) * 1.03


def _steps(case):
    """Modular multiplications of the walk: one per n (prime n for n#, composite n for n!/n#), per candidate."""
    n = case["nmax"] - case["nmin"]
    primes = n / math.log(case["nmax"])
    per = {1: n, 2: primes, 4: n - primes, 5: 2 * n - primes}[case["mode"]]
    return _candidates(case) * per


def _hits(case):
    """Expected hits: a residue is +-1 with probability 2/p."""
    return 2 * _steps(case) / case["pmin"]


def _seconds(case):
    """A rough upper estimate, to keep drawn cases no dearer than the largest listed one."""
    rate = 2e12 if case["pmax"] <= SPLIT32 else 1e12 if case["pmax"] <= LAZY_END else 5e11
    setup = _candidates(case) * case["nmax"] * (3e-15 if case["pmax"] <= SPLIT32 else 6e-15)
    if case["pmax"] > LAZY_END:
        setup *= 20
    check = _hits(case) * case["nmax"] / (1e11 if case["verify"] == "device" else 4e9)
    return _steps(case) / rate + setup + check + case["nmax"] * 3e-9


def draw(rng):
    kind = rng.random()
    if kind < 0.1:
        return {"kind": "batch", "count": rng.randint(3, 40), "n0": _log(rng, 10**4, 10**7),
                "nlen": _log(rng, 10**4, 2 * 10**5), "plen": _log(rng, 10**6, 10**7)}
    if kind < 0.2:
        nmax = _log(rng, 10**4, 3 * 10**5)
        pmin = _log(rng, 5 * 10**5, 10**7)
        return {"kind": "verify", "mode": rng.choice((1, 2, 4, 5)), "nmin": 101, "nmax": nmax, "pmin": pmin,
                "pmax": pmin + _log(rng, 5 * 10**4, 5 * 10**5)}
    while True:
        nmin = _log(rng, 101, 10**7)
        nmax = nmin + _log(rng, 1000, 10**6)
        pmin = _log(rng, 10**6, 2**64 - 2 * 10**8)
        case = {"kind": "search", "mode": rng.choice((1, 2, 4, 5)), "nmin": nmin, "nmax": nmax, "pmin": pmin,
                "pmax": pmin + _log(rng, 10**5, 10**8), "verify": "device" if nmax > 10**6 else "cpu"}
        if rng.random() < 0.15:
            case["kind"] = "segments"
            case["parts"] = rng.randint(2, 6)
            case["verify"] = "cpu"
        if _seconds(case) <= 0.7:
            if case["kind"] == "segments":
                del case["verify"]
            return case


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def _bounds(case, seed):
    """The seed's p range: the case's length, moved by less than that length."""
    span = case["pmax"] - case["pmin"]
    lo = case["pmin"] + random.Random(seed).randrange(1, span)
    return lo, lo + span


def prepare(case, seed):
    ctx = pfc.Context(0)
    state = {"case": case, "ctx": ctx, "threads": os.cpu_count() or 2}
    if case["kind"] == "batch":
        state["searches"] = [s.astuple() for s in serving.mixed_jobs(
            case["count"], seed=seed, n_len=(1e3, case["nlen"]), n0=(101, case["n0"]), p_len=(1e5, case["plen"]))]
        return state
    lo, hi = state["p"] = _bounds(case, seed)
    if case["kind"] == "segments":
        state["job"] = pfc.Job(ctx, case["mode"], case["nmin"], case["nmax"], lo, hi)
        state["done"] = 0, 0
    elif case["kind"] == "verify":
        with pfc.Job(ctx, case["mode"], case["nmin"], case["nmax"], lo, hi) as job:
            hits = job.run()
        state["hits"] = hits[np.lexsort((hits["nc"], hits["type"], hits["p"]))]
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        with pfc.Batch(state["ctx"]) as batch:
            ids = [batch.submit(*s) for s in state["searches"]]
            batch.run()
            out, sums = [], []
            for i, s in zip(ids, state["searches"]):
                st = batch.status(i)
                sums.append((st.status, st.term_checksum, st.primecount, st.pairs))
                out.append(pfc.finalize(s[0], s[2], batch.hits(i), verify="device", ctx=state["ctx"]))
                batch.release(i)
        return {"totals": np.array(sums, dtype=np.uint64).view(np.int64), **_factors(case, [k for k, _ in out]),
                "addends": np.array([a for _, a in out], dtype=np.uint64).view(np.int64)}
    if case["kind"] == "verify":
        bad = pfc.verify_factors(state["ctx"], case["mode"], case["nmax"], state["hits"])
        room = np.zeros(_room(case), dtype=bool)
        room[:len(bad)] = bad
        return {"bad": room, **_factors(case, [state["hits"]])}
    lo, hi = state["p"]
    if case["kind"] == "segments":
        job, parts = state["job"], []
        step = -(-(hi - lo) // case["parts"])
        while lo < hi:
            end = min(job.segment_end(lo), lo + step, hi)
            job.segment(lo, end)
            parts.append(pfc.finalize(case["mode"], case["nmax"], job.drain_hits(), threads=state["threads"]))
            lo = end
        totals = job.totals()   # of the job since its start: this pass's part is returned
        (t0, c0), state["done"] = state["done"], totals
        sums = [(totals[0] - t0 + sum(a for _, a in parts)) % 2**64, totals[1] - c0]
        return {"totals": np.array(sums, dtype=np.uint64).view(np.int64), **_factors(case, [k for k, _ in parts])}
    r = pfc.sieve(case["mode"], case["nmin"], case["nmax"], lo, hi, threads=state["threads"],
                  verify="device" if case["verify"] == "device" else True, ctx=state["ctx"])
    return _result(case, r.checksum, r.primecount, r.pairs, r.factors)


def _result(case, checksum, primecount, pairs, factors):
    return {"totals": np.array([checksum, primecount, pairs], dtype=np.uint64).view(np.int64),
            **_factors(case, [factors])}


def _room(case):
    """Records of the factor list as returned: the list, then zeros (p ranges of one length differ in their hits)."""
    return 2048 * case["count"] if case["kind"] == "batch" else int(2 * _hits(case)) + 256


def _factors(case, parts):
    f = np.zeros(_room(case), dtype=pfc.FACTOR_DTYPE)
    got = np.concatenate(parts)
    f[:len(got)] = got
    return {"p": f["p"].view(np.int64), "nc": f["nc"], "type": f["type"]}


def work(case):
    """Two operations (a product and its reduction) per modular multiplication; candidates written once."""
    if case["kind"] == "batch":   # the mix's mean lengths
        def mean(lo, hi):
            return (hi - lo) / math.log(hi / lo)
        cands = case["count"] * mean(1e5, case["plen"]) / 31
        return {"bytes": 8 * cands, "flops": 2 * cands * mean(1e3, case["nlen"]) * 0.65}
    if case["kind"] == "verify":
        return {"bytes": 17 * _hits(case), "flops": 2 * _hits(case) * case["nmax"] / 2}
    width = 4 if case["pmax"] <= SPLIT32 else 8
    return {"bytes": width * _candidates(case) + 16 * _hits(case), "flops": 2 * _steps(case)}


def exact(case, seed):
    """The search's definition in 64-bit numpy (p below 2^31), where that is quick."""
    if case["kind"] != "search" or case["mode"] != 1 or case["pmax"] * 2 > 2**31 or \
            _candidates(case) * case["nmax"] > 5e8:
        return None
    lo, hi = _bounds(case, seed)
    odd = np.arange(max(lo | 1, 115), hi, 2, dtype=np.int64)
    small = [q for q in range(3, 114) if all(q % d for d in range(2, q))]
    for q in small:
        odd = odd[odd % q != 0]
    p = np.array([x for x in odd.tolist() if _sprp2(x)], dtype=np.int64)
    r = np.ones_like(p)
    hits, terms = [], 0
    for n in range(2, case["nmax"]):
        r = r * n % p
        if n >= case["nmin"]:
            hits += [(int(q), -n) for q in p[r == 1]] + [(int(q), n) for q in p[r == p - 1]]
    hits = sorted((h for h in hits if _prime(h[0])), key=lambda h: (h[0], abs(h[1])))
    for q, s in zip(p.tolist(), r.tolist()):   # the checksum: final residue and last n in Montgomery form, R = 2^64
        terms += (s << 64) % q + ((case["nmax"] - 1) << 64) % q
    checksum = (terms + sum(abs(n) + (1 if n > 0 else -1) for _, n in hits)) % 2**64
    f = np.array([(q, n, 0) for q, n in hits], dtype=pfc.FACTOR_DTYPE)
    return _result(case, checksum, len(p), len(p) * (case["nmax"] - case["nmin"]), f)


def _sprp2(x):
    d, t = x - 1, 0
    while d % 2 == 0:
        d, t = d // 2, t + 1
    a = pow(2, d, x)
    return a in (1, x - 1) or any((a := a * a % x) == x - 1 for _ in range(t - 1))


def _prime(x):
    return all(x % d for d in range(3, math.isqrt(x) + 1, 2))
