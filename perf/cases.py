"""The workloads this engine is timed on: full transforms, partial outputs and
mixed batches, each through the package's public calls.

A case is a dict of plain values.  Full transforms: field, log_n, batch,
inverse.  Partial outputs: field, log_n, pattern (prefix / strided / random)
and count.  Mixed batches: the number of requests and the seed they are drawn
from.  Domains, batches and the planner are made once per process and kept,
as a program that runs many transforms keeps them; every state holds its own
inputs and output buffers.
"""
from __future__ import annotations

import functools
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "omr-ntt_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import omr_ntt  # noqa: E402
from omr_ntt import batch as mixed  # noqa: E402
from omr_ntt import planner  # noqa: E402
from omr_ntt.fields import Goldilocks, field_by_name  # noqa: E402

_PATTERN = {"prefix": omr_ntt.PREFIX, "strided": omr_ntt.STRIDED, "random": omr_ntt.INDICES}


def _full(name, field, log_n, batch=1, inverse=False):
    return {"name": name, "kind": "full", "field": field, "log_n": log_n, "batch": batch, "inverse": inverse}


def _partial(name, field, log_n, pattern, count):
    return {"name": name, "kind": "partial", "field": field, "log_n": log_n, "pattern": pattern, "count": count}


def listed():
    return [
        # one short transform alone: launch and latency bound (the smoke size)
        _full("gl_fwd_2e12", "Goldilocks", 12),
        # the crate's plain radix-2 benchmark size, one transform
        _full("bb_fwd_2e16", "BabyBear", 16),
        # a medium single transform, and a batch of an odd count in one of
        # the two other 31/32-bit fields
        _full("bb_fwd_2e20", "BabyBear", 20),
        _full("kb_inv_2e18x5", "KoalaBear", 18, batch=5, inverse=True),
        _full("gl_inv_2e22", "Goldilocks", 22, inverse=True),
        # the headline size in both main fields
        _full("bb_fwd_2e24", "BabyBear", 24),
        _full("gl_fwd_2e24", "Goldilocks", 24),
        # many columns of a proof trace at once, back to coefficients
        _full("bb_inv_2e20x64", "BabyBear", 20, batch=64, inverse=True),
        # partial outputs of one 2^22 transform: the first 2s = 100 (the
        # crate's profiling example has s = 50), a coset, and a random set
        _partial("bb_2e22_prefix_100", "BabyBear", 22, "prefix", 100),
        _partial("bb_2e22_strided_2e12", "BabyBear", 22, "strided", 1 << 12),
        _partial("gl_2e22_random_2e8", "Goldilocks", 22, "random", 1 << 8),
        # a server's queue: requests of 2^10..2^20 points in two fields and
        # both directions, a quarter of them with partial outputs, one launch
        {"name": "mixed_4096", "kind": "mixed", "requests": 4096, "request_seed": 2024},
    ]


def draw(rng):
    kind = rng.choice(["full", "full", "full", "partial", "partial", "mixed"])
    if kind == "full":
        field = rng.choice(["BabyBear", "BabyBear", "Goldilocks", "Goldilocks", "KoalaBear", "TeddyBear"])
        log_n = rng.randint(10, 24)
        most = min(512, (1 << 26) >> log_n)
        batch = 1 if rng.random() < 0.5 else int(round(most ** rng.random()))
        return {"kind": kind, "field": field, "log_n": log_n, "batch": max(1, batch),
                "inverse": rng.random() < 0.5}
    if kind == "partial":
        log_n = rng.randint(16, 24)
        pattern = rng.choice(["prefix", "strided", "random"])
        log_c = rng.uniform(4, min(16, log_n - 2))
        count = 1 << int(log_c) if pattern == "strided" else int(2 ** log_c)
        return {"kind": kind, "field": rng.choice(["BabyBear", "Goldilocks"]), "log_n": log_n,
                "pattern": pattern, "count": count}
    return {"kind": kind, "requests": int(2 ** rng.uniform(6, 11)), "request_seed": rng.randint(1, 10000)}


# ---------------------------------------------------------------- kept handles


@functools.lru_cache(maxsize=None)
def _planner():
    return planner.install_default()


@functools.lru_cache(maxsize=None)
def _domain(field_name, log_n):
    _planner()
    return omr_ntt.NttDomain(field_by_name(field_name), 1 << log_n)


@functools.lru_cache(maxsize=2)
def _batch(requests, request_seed):
    _planner()
    reqs = mixed.mixed_requests(request_seed, count=requests)
    in_bytes, out_bytes = mixed.layout(reqs)
    return mixed.Batch(reqs), in_bytes, out_bytes


# ---------------------------------------------------------------- inputs


def _words(field, count, gen, out=None):
    """count uniform canonical words (the words' bits in a signed tensor)."""
    if field.word_bytes == 4:
        x = torch.randint(0, field.p, (count,), dtype=torch.int64, device="cuda", generator=gen)
        x = x.to(torch.int32)
    else:  # p = 2^64 - 2^32 + 1: a high half below 2^32 - 1 is canonical with any low half
        hi = torch.randint(-(1 << 31), (1 << 31) - 1, (count,), dtype=torch.int64, device="cuda", generator=gen)
        hi = hi + (hi >= -1)  # every 32-bit high half but 0xffffffff
        x = torch.randint(0, 1 << 32, (count,), dtype=torch.int64, device="cuda", generator=gen)
        x += hi << 32
    if out is None:
        return x
    out.copy_(x)
    return out


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["kind"] == "mixed":
        handle, in_bytes, out_bytes = _batch(case["requests"], case["request_seed"])
        # BabyBear words everywhere, then the Goldilocks requests' own words
        x = torch.randint(0, 0x78000001, ((in_bytes + 7) // 8 * 2,), dtype=torch.int32, device="cuda",
                          generator=gen)
        wide = x.view(torch.int64)
        for r in handle.reqs:
            if r.field is Goldilocks:
                at = r.in_off // 8
                _words(Goldilocks, r.n, gen, wide[at:at + r.n])
        out = torch.zeros((out_bytes + 3) // 4, dtype=torch.int32, device="cuda")
        return {"case": case, "batch": handle, "x": x, "out": out}
    field = field_by_name(case["field"])
    domain = _domain(case["field"], case["log_n"])
    if case["kind"] == "full":
        x = _words(field, case["batch"] << case["log_n"], gen)
        return {"case": case, "domain": domain, "x": x, "out": torch.empty_like(x)}
    x = _words(field, 1 << case["log_n"], gen)
    indices = None
    if case["pattern"] == "random":
        idx = omr_ntt.random_indices(1 << case["log_n"], case["count"], int(seed))
        indices = torch.from_numpy(idx.view(np.int32)).cuda()
    out = torch.empty(case["count"], dtype=x.dtype, device="cuda")
    return {"case": case, "domain": domain, "x": x, "indices": indices, "out": out}


def run(state):
    case = state["case"]
    if case["kind"] == "full":
        call = omr_ntt.inverse if case["inverse"] else omr_ntt.forward
        return call(state["domain"], state["x"], out=state["out"], batch=case["batch"])
    if case["kind"] == "partial":
        return omr_ntt.partial(state["domain"], state["x"], _PATTERN[case["pattern"]], case["count"],
                               indices=state["indices"], out=state["out"])
    state["batch"].run(state["x"].data_ptr(), state["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    return state["out"]


def work(case):
    """Each input word read once, each output word written once; operations
    are integer ones: N/2 log2 N butterflies of a modular product, sum and
    difference for a full transform, one addition per input for the rest."""
    if case["kind"] == "full":
        n, w = 1 << case["log_n"], field_by_name(case["field"]).word_bytes
        return {"bytes": 2 * n * case["batch"] * w, "flops": 1.5 * n * case["log_n"] * case["batch"]}
    if case["kind"] == "partial":
        n, w = 1 << case["log_n"], field_by_name(case["field"]).word_bytes
        index_bytes = 4 * case["count"] if case["pattern"] == "random" else 0
        return {"bytes": (n + case["count"]) * w + index_bytes, "flops": float(n)}
    total = {"bytes": 0, "flops": 0.0}
    for r in _requests(case["requests"], case["request_seed"]):
        n, w, outs, log_n, index_bytes = r
        total["bytes"] += (n + outs) * w + index_bytes
        total["flops"] += 1.5 * n * log_n
    return total


@functools.lru_cache(maxsize=8)
def _requests(requests, request_seed):
    return [(r.n, r.field.word_bytes, r.out_words, r.log_n, 0 if r.indices is None else 4 * len(r.indices))
            for r in mixed.mixed_requests(request_seed, count=requests)]


# ---------------------------------------------------------------- exact values


def _mul(a, b, p):
    """a b mod p on uint64 arrays of canonical words."""
    if p < 1 << 32:
        return a * b % np.uint64(p)
    m, s = np.uint64(0xffffffff), np.uint64(32)
    a0, a1, b0, b1 = a & m, a >> s, b & m, b >> s
    low, mid0, mid1, high = a0 * b0, a0 * b1, a1 * b0, a1 * b1
    mid = (low >> s) + (mid0 & m) + (mid1 & m)
    high = high + (mid0 >> s) + (mid1 >> s) + (mid >> s)
    low = (low & m) | (mid << s)
    # 2^64 = 2^32 - 1 and 2^96 = -1 (mod p)
    r = _sub(low % np.uint64(p), high >> s, p)
    return _add(r, (high & m) * m % np.uint64(p), p)


def _add(a, b, p):
    b = np.uint64(p) - b
    return np.where(a >= b, a - b, a - b + np.uint64(p))


def _sub(a, b, p):
    return np.where(a >= b, a - b, a - b + np.uint64(p))


def exact(case, seed):
    """The same outputs from a plain radix-2 transform in numpy."""
    if case["kind"] == "mixed" or (case.get("batch", 1) << case["log_n"]) > 1 << 20:
        return None
    field, log_n = field_by_name(case["field"]), case["log_n"]
    n, p = 1 << log_n, field.p
    state = prepare(case, seed)
    x = state["x"].cpu().numpy()
    x = x.view(np.uint32 if field.word_bytes == 4 else np.uint64).astype(np.uint64).reshape(-1, n)
    w = field.root_of_unity(log_n)
    if case.get("inverse"):
        w = pow(w, p - 2, p)
    root = np.ones(1, dtype=np.uint64)
    for i in range(log_n - 1):  # powers of w by doubling
        root = np.concatenate([root, _mul(root, np.full_like(root, pow(w, 1 << i, p)), p)])
    with np.errstate(over="ignore"):
        for i in range(log_n):  # decimation in frequency, outputs bit-reversed
            half = n >> (i + 1)
            v = x.reshape(-1, 2, half)
            a, b = v[:, 0], v[:, 1]
            t = np.broadcast_to(root[:: 1 << i][:half], a.shape)
            x = np.stack([_add(a, b, p), _mul(_sub(a, b, p), t, p)], axis=1).reshape(-1, n)
        order = np.zeros(1, dtype=np.int64)
        for i in range(log_n):
            order = np.concatenate([2 * order, 2 * order + 1])
        x = x[:, order]
        if case.get("inverse"):
            x = _mul(x, np.full_like(x, pow(n, p - 2, p)), p)
    x = x.reshape(-1)
    if case["kind"] == "partial":
        k = np.arange(case["count"])
        if case["pattern"] == "strided":
            k = k * (n // case["count"])
        elif case["pattern"] == "random":
            k = state["indices"].cpu().numpy().view(np.uint32)
        x = x[k]
    x = x.astype(np.uint32).view(np.int32) if field.word_bytes == 4 else x.view(np.int64)
    return torch.from_numpy(np.ascontiguousarray(x))
