"""Exhaustive tuning of partial outputs into a planner database file.

    python -m omr_ntt.tune_partial              # writes omr-ntt_gb300/data/planner_partial.db
    python -m omr_ntt.tune_partial --out PATH --min-log 16 --max-log 24

For BabyBear and Goldilocks, log2 N in [min-log, max-log], prefixes and index
sets of up to 2^9 outputs (2^11 from 2^18 on) and strided sets of 2^13 to 2^16,
the exhaustive autotuner (omr_ntt_tune_point) times every plan.  An entry serves
every count in (2^(k-1), 2^k], so a plan is judged at both ends of that range, by
its times over the fastest there; the built-in rule's choice is kept where it is
within 3% of the best, which is what short calls' times are good to.
`planner.install_default()` loads the file.  These are the counts at which the
learned selector takes line lengths and strategies up to a third slower than the
best; it decides the other counts.  (Three entries of the shipped file, Goldilocks
2^21 with 65..128 random indices, 2^22 with a prefix of 257..512 and 2^24 with 2^16
strided outputs, are taken out: their calls on data in L2 took 4-7% longer than
with the selector's choice.)
"""
from __future__ import annotations

import argparse
import ctypes
import json
import os
import time

import numpy as np

from . import planner as P
from ._lib import check, lib
from .fields import BabyBear, Goldilocks



def log_counts(log_n: int, pattern: str):
    if pattern == "strided":
        return range(13, min(16, log_n - 2) + 1)
    return range((11 if log_n >= 18 else 9) + 1)


def shapes(min_log: int, max_log: int):
    for f in (BabyBear, Goldilocks):
        for log_n in range(min_log, max_log + 1):
            for pattern in ("contiguous", "strided", "random"):
                for k in log_counts(log_n, pattern):
                    yield f, log_n, pattern, k


def rule_candidate(f, log_n, pattern, k):
    """(strategy, param) that the built-in rule takes for 2^k outputs; its lines lie between the ranges."""
    p = {"field": f.id, "log_n": log_n, "log_s": k, "pattern": pattern, "batch": 1}
    s, q = ctypes.c_int(), ctypes.c_int()
    ok = lib().omr_ntt_plan_class_candidate(f.id, log_n, P.PATTERN_ID[pattern], 1 << k, P.heuristic_class(p),
                                            ctypes.byref(s), ctypes.byref(q))
    return (s.value, q.value) if ok == 1 else None


def tune_counts(f, log_n, pattern, counts, reps):
    """Candidates (the same for all `counts` of a bucket) and their mean time over the fastest."""
    pat, score, cands = P.PATTERN_ID[pattern], 0.0, None
    for c in counts:
        n = lib().omr_ntt_candidates(f.id, log_n, pat, c, None, None, 0)
        st, pa, ms = (ctypes.c_int * n)(), (ctypes.c_int * n)(), (ctypes.c_float * n)()
        lib().omr_ntt_candidates(f.id, log_n, pat, c, st, pa, n)
        rc = lib().omr_ntt_tune_point(f.id, log_n, 1, pat, c, reps, log_n * 1000 + c, ms, n)
        if rc < 0:
            check(rc)
        t = np.array(list(ms), dtype=np.float64)
        assert cands is None or cands == list(zip(list(st), list(pa)))
        cands = list(zip(list(st), list(pa)))
        score = score + t / t.min() / len(counts)
    return cands, score


def main(argv=None):
    ap = argparse.ArgumentParser()
    ap.add_argument("--out", default=os.path.join(P.DATA_DIR, "planner_partial.db"))
    ap.add_argument("--min-log", type=int, default=16)
    ap.add_argument("--max-log", type=int, default=24)
    ap.add_argument("--reps", type=int, default=5)
    a = ap.parse_args(argv)
    check(lib().omr_ntt_planner_clear())
    t0 = time.time()
    entries = 0
    for f, log_n, pattern, k in shapes(a.min_log, a.max_log):
        top = 1 << k
        counts = [top] if pattern == "strided" or k < 2 else [top // 2 + 1, top]
        cands, score = tune_counts(f, log_n, pattern, counts, a.reps)
        i = int(np.argmin(score))
        rule = rule_candidate(f, log_n, pattern, k)
        if rule in cands and score[cands.index(rule)] <= 1.03 * score[i]:
            i = cands.index(rule)
        check(lib().omr_ntt_planner_set(f.id, log_n, 1, P.PATTERN_ID[pattern], top, *cands[i]))
        entries += 1
    check(lib().omr_ntt_planner_save(a.out.encode()))
    print(json.dumps({"entries": entries, "seconds": round(time.time() - t0, 1), "out": a.out}))


if __name__ == "__main__":
    main()
