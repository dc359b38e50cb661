"""The built-in plan rule on batches (no GPU): on both sides of the lines where
another plan takes over, the plan class of the Python mirror and the passes the
library runs for it.  (KoalaBear and TeddyBear: the learned selector leaves them
to the rule.)"""
import ctypes

import pytest

import omr_ntt
from omr_ntt import _lib
from omr_ntt import planner as P
from omr_ntt.fields import KoalaBear, TeddyBear

L = _lib.lib()

POINTS = [(KoalaBear, 10, 128, "32x32 cluster"), (KoalaBear, 10, 129, "32x32 slab"), (KoalaBear, 11, 100, "64x32 cluster"),
          (KoalaBear, 11, 400, "64x32 slab"), (TeddyBear, 11, 400, "64x32 slab"), (KoalaBear, 12, 256, "64x64 cluster"), (KoalaBear, 12, 304, "64x64 slab"),
          (KoalaBear, 12, 305, "64x64 cluster"), (KoalaBear, 12, 512, "64x64 slab"), (TeddyBear, 12, 304, "64x64 cluster"),
          (KoalaBear, 12, 400, "64x64 cluster"),
          (KoalaBear, 16, 7, "256x256 tma2cta"), (KoalaBear, 16, 8, "256x256 cluster"),
          (TeddyBear, 16, 40, "256x256 cluster"), (KoalaBear, 16, 41, "256x256 wide"),
          (KoalaBear, 18, 24, "512x512 slab"), (TeddyBear, 18, 24, "512x512 tma2cta"), (TeddyBear, 18, 40, "512x512 slab"),
          (KoalaBear, 19, 4, "1024x512 slab"), (TeddyBear, 19, 4, "1024x512 tma2cta"), (TeddyBear, 19, 16, "1024x512 slab"),
          (KoalaBear, 20, 3, "1024x1024 slab"), (TeddyBear, 20, 3, "1024x1024 tma2cta"),
          (TeddyBear, 20, 16, "1024x1024 slab"), (KoalaBear, 21, 4, "4096x512 slab"), (TeddyBear, 21, 1, "4096x512 slab"),
          (TeddyBear, 21, 5, "2048x1024 tma2cta"), (TeddyBear, 21, 6, "128x128x128 slab")]


def passes(field, log_n, plan, batch):
    rec = (ctypes.c_uint64 * 64)()
    n = L.omr_ntt_plan_passes(field.id, log_n, plan, batch, rec, 4)
    return [list(rec[16 * i:16 * i + 16]) for i in range(n)]


@pytest.mark.parametrize("field,log_n,batch,plan", POINTS, ids=lambda v: str(getattr(v, "name", v)).replace(" ", "-"))
def test_rule(field, log_n, batch, plan):
    p = {"field": field.id, "log_n": log_n, "log_s": log_n, "pattern": "contiguous", "batch": batch}
    s, i = ctypes.c_int(), ctypes.c_int()
    assert L.omr_ntt_plan_class_candidate(field.id, log_n, 0, 1 << log_n, P.heuristic_class(p), ctypes.byref(s),
                                          ctypes.byref(i)) == 1
    assert omr_ntt.plan_describe(field, log_n, i.value) == "four-step " + plan
    L.omr_ntt_planner_clear()
    assert passes(field, log_n, -1, batch) == passes(field, log_n, i.value, batch)


@pytest.mark.parametrize("field,log_n,pattern,log_s,plan",
                         [(KoalaBear, 21, "contiguous", 16, "2048x1024 slab"), (KoalaBear, 21, "random", 15, "2048x1024 slab"),
                          (KoalaBear, 21, "random", 16, "4096x512 slab"), (TeddyBear, 21, "contiguous", 16, "2048x1024 tma2cta"),
                          (TeddyBear, 21, "random", 13, "2048x1024 tma2cta"), (TeddyBear, 21, "random", 16, "2048x1024 tma2cta"),
                          (TeddyBear, 20, "contiguous", 16, "1024x1024 tma2cta")],
                         ids=lambda v: str(getattr(v, "name", v)).replace(" ", "-"))
def test_plan_behind_a_gather(field, log_n, pattern, log_s, plan):
    p = {"field": field.id, "log_n": log_n, "log_s": log_s, "pattern": pattern, "batch": 1}
    s, i = ctypes.c_int(), ctypes.c_int()
    assert L.omr_ntt_plan_class_candidate(field.id, log_n, P.PATTERN_ID[pattern], 1 << log_s, P.heuristic_class(p),
                                          ctypes.byref(s), ctypes.byref(i)) == 1
    assert s.value == 3 and omr_ntt.plan_describe(field, log_n, i.value) == "four-step " + plan
