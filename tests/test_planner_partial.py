"""The shipped plans of partial outputs (no GPU): all are valid for their
largest count, and over the committed timings they are no
worse than the learned selector, which ranked the decomposition of 257..512
outputs first at 2^16..2^18 where a transform and gather take three quarters of
its time."""
import ctypes
import json
import os

import numpy as np

from omr_ntt import _lib
from omr_ntt import planner as P
from omr_ntt.tune_partial import shapes
from oracle import mlp_ref

L = _lib.lib()
GATHER = 3


def get(field, log_n, pattern, k):
    s, q = ctypes.c_int(), ctypes.c_int()
    ok = L.omr_ntt_planner_get(field, log_n, 1, P.PATTERN_ID[pattern], 1 << k, ctypes.byref(s), ctypes.byref(q))
    return (s.value, q.value) if ok else None


def load():
    L.omr_ntt_planner_clear()
    for db in (P.DEFAULT_DB, P.DEFAULT_PARTIAL_DB):
        assert L.omr_ntt_planner_load(db.encode()) > 0


def test_plans_are_valid():
    load()
    try:
        for f, log_n, pattern, k in shapes(16, 24):
            p = {"field": f.id, "log_n": log_n, "log_s": k, "pattern": pattern, "batch": 1}
            c = get(f.id, log_n, pattern, k)
            assert c is None or c in P.candidates(p), p
            if pattern != "strided" and log_n <= 18 and k == 9:
                assert c and c[0] == GATHER, p
    finally:
        L.omr_ntt_planner_clear()


def test_no_worse_than_the_selector():
    z = np.load(os.path.join(P.DATA_DIR, "planner_dataset.npz"))
    X, T, best, pts = z["X"], z["T"].astype(np.float64), z["best"].astype(np.float64), json.loads(str(z["points"]))
    params, _ = P.load_params(os.path.join(P.DATA_DIR, "planner_mlp.npz"))
    pred = mlp_ref.forward(params, X, P.N_FEATURES, P.N_HIDDEN, T.shape[1])
    net = P.regret(T, best, P.choose(pred, T))
    load()
    try:
        shipped, selector = [], []
        for i, p in enumerate(pts):
            c = get(p["field"], p["log_n"], p["pattern"], p["log_s"]) if p["log_s"] < p["log_n"] else None
            if p["batch"] > 1 or c is None:
                continue
            cands, where = P.candidates(p), P.class_map(p)
            j = [k for k, w in enumerate(where) if w >= 0 and cands[w] == c]
            if j:  # (a plan outside the classes has no committed time)
                shipped.append(T[i, j[0]] / best[i] - 1)
                selector.append(net[i])
        assert len(shipped) > 50
        assert np.mean(shipped) <= np.mean(selector)
    finally:
        L.omr_ntt_planner_clear()
