"""The engine's work as its users have it done, in cases that can be timed and compared.

A case is one of four kinds, each through the public entry points of mersenne2gpu_gb300:

  advance  a lone LL / PRP / PRP3 test taken from one checkpoint to the next: the residue's digits go in
           (Engine.set_digits), one report batch of squarings runs (Engine.iterate), the canonical digits come out
           (Engine.digits).  This is what the command line tool does between two checkpoints, and what a host
           program does that owns the residue.  Host buffers are pinned, as a program that checkpoints often has them.
  gerbicz  the same for a PRP chain under the Gerbicz error check: two check blocks, the verification, and the
           verified state.
  batch    many independent PRP tests in one call (batch_run), every test capped to the same number of squarings.
  serve    the continuous-batching server: requests submitted, stepped until all of them are done, results polled.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import mersenne2gpu_gb300 as m2
from mersenne2gpu_gb300.serve import Server

MODES = {"ll": m2.MODE_LL, "prp": m2.MODE_PRP, "prp3": m2.MODE_PRP3}
# exponent range of the lone tests: the smallest request of the serving workload up to the largest exponent of n = 2^22
LONE = (1000, 142606333)
SERVE = (1000, 18874367)
BATCH = (3, 159739)
# no drawn case costs more than this many digit-squarings times levels: the largest listed case's
MOST = 500 * (1 << 22) * 21


def listed():
    return [
        # a small exponent, its state checked every 1000 squarings: one transform far too small for the GPU, all latency
        {"name": "prp 9941", "kind": "advance", "p": 9941, "mode": "prp", "iters": 1000, "fields": "dual"},
        # mid-size lone tests, a full run of which takes seconds (n = 4096 and 8192)
        {"name": "prp 132049", "kind": "advance", "p": 132049, "mode": "prp", "iters": 1000, "fields": "dual"},
        {"name": "ll 216091", "kind": "advance", "p": 216091, "mode": "ll", "iters": 1000, "fields": "dual"},
        # lone tests of minutes to hours (n = 2^16, 2^18, 2^19)
        {"name": "ll 1257787", "kind": "advance", "p": 1257787, "mode": "ll", "iters": 1000, "fields": "dual"},
        {"name": "prp3 6972593", "kind": "advance", "p": 6972593, "mode": "prp3", "iters": 1000, "fields": "dual"},
        {"name": "prp 13466917", "kind": "advance", "p": 13466917, "mode": "prp", "iters": 1000, "fields": "dual"},
        # the headline exponent (n = 2^21), with both fields and in the GF(P61^2)-only layout (n = 2^22)
        {"name": "prp 57885161", "kind": "advance", "p": 57885161, "mode": "prp", "iters": 1000, "fields": "dual"},
        {"name": "prp 57885161 gf61", "kind": "advance", "p": 57885161, "mode": "prp", "iters": 500, "fields": "gf61"},
        # the largest transform in ordinary use (n = 2^22)
        {"name": "ll 115640321", "kind": "advance", "p": 115640321, "mode": "ll", "iters": 500, "fields": "dual"},
        # a long PRP run that checks itself (n = 2^20)
        {"name": "gerbicz 24036583", "kind": "gerbicz", "p": 24036583, "block": 200},
        # a sweep of small exponents in one call (n = 8 ... 4096)
        {"name": "batch 1024", "kind": "batch", "tests": 1024, "iters": 500},
        # requests of mixed sizes sharing the GPU (n = 32 ... 2^19)
        {"name": "serve 64", "kind": "serve", "requests": 64, "iters": 500, "quantum": 250},
    ]


def _is_prime(n):
    if n < 2:
        return False
    small = (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37)
    for q in small:
        if n % q == 0:
            return n == q
    d, s = n - 1, 0
    while d % 2 == 0:
        d, s = d // 2, s + 1
    for a in small[:4]:   # enough below 3.2e9
        x = pow(a, d, n)
        if x in (1, n - 1):
            continue
        for _ in range(s - 1):
            x = x * x % n
            if x == n - 1:
                break
        else:
            return False
    return True


def _prime_near(x, lo, hi):
    """The first prime from x on, or the last one up to hi."""
    x = min(max(int(x), lo), hi)
    up = x
    while up <= hi and not _is_prime(up):
        up += 1
    if up <= hi:
        return up
    while not _is_prime(x):
        x -= 1
    return x


def _log_uniform(rng, lo, hi):
    return lo * math.exp(rng.random() * math.log(hi / lo))


def _log2_digits(p, fields="dual"):
    """log2 of the transform length of exponent p (the size rule of m2_layout)."""
    bound, ln = (61 if fields == "gf61" else 92), 3
    while ln + 2 * ((p >> ln) + 1) >= bound:
        ln += 1
    return ln


def draw(rng):
    kind = rng.choices(("advance", "gerbicz", "batch", "serve"), (14, 3, 2, 2))[0]
    if kind == "batch":
        return {"kind": "batch", "tests": int(_log_uniform(rng, 64, 1024)), "iters": rng.randint(100, 500)}
    if kind == "serve":
        return {"kind": "serve", "requests": rng.randint(8, 64), "iters": rng.randint(100, 500), "quantum": rng.randint(100, 300)}
    if kind == "gerbicz":
        p = _prime_near(_log_uniform(rng, 10000, 57885161), *LONE)
        return {"kind": "gerbicz", "p": p, "block": rng.randint(20, 200)}
    fields = rng.choices(("dual", "gf61"), (6, 1))[0]
    p = _prime_near(_log_uniform(rng, LONE[0], 57885161 if fields == "gf61" else LONE[1]), *LONE)
    ln = _log2_digits(p, fields)
    iters = min(int(_log_uniform(rng, 30, 1000)), MOST // ((1 << ln) * (ln - 1)))
    return {"kind": "advance", "p": p, "mode": rng.choice(("prp", "prp", "ll", "prp3")), "iters": iters, "fields": fields}


def _digits(p, fields, seed):
    """A residue in mid-run: n uniform digits below their widths."""
    _, n, w = m2.layout(p, m2.FIELDS_GF61 if fields == "gf61" else m2.FIELDS_DUAL)
    raw = np.random.default_rng(seed).integers(0, 1 << 62, n, dtype=np.uint64)
    return raw & ((np.uint64(1) << w.astype(np.uint64)) - np.uint64(1))


def _exponents(case, seed):
    rng = random.Random(seed)
    if case["kind"] == "batch":
        return [_prime_near(rng.randint(*BATCH), *BATCH) for _ in range(case["tests"])]
    return [_prime_near(_log_uniform(rng, *SERVE), *SERVE) for _ in range(case["requests"])]


class _Lone:
    """One engine, the digits that it starts from and the buffer that it ends in."""

    def __init__(self, case, seed):
        fields = case.get("fields", "dual")
        start = _digits(case["p"], fields, seed)
        # the pinned host tensors (uint64 digits are below 2^62: int64 holds them)
        self.t_in = torch.from_numpy(start.view(np.int64)).pin_memory()
        self.t_out = torch.empty_like(self.t_in).pin_memory()
        self.start = self.t_in.numpy().view(np.uint64)
        self.out = self.t_out.numpy().view(np.uint64)
        self.eng = m2.Engine(case["p"], MODES[case.get("mode", "prp")],
                             fields=m2.FIELDS_GF61 if fields == "gf61" else m2.FIELDS_DUAL)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("advance", "gerbicz"):
        return case, _Lone(case, seed)
    return case, _exponents(case, seed)


def run(state):
    case, held = state
    kind = case["kind"]
    if kind == "advance":
        held.eng.set_digits(held.start, 0)
        held.eng.iterate(case["iters"])
        return held.eng.digits(held.out).view(np.int64)
    if kind == "gerbicz":
        held.eng.set_digits(held.start, 0)
        with m2.Gec(held.eng, case["block"]) as g:
            g.iterate(2 * case["block"])
            good = g.check()
            digits, at = g.verified()
        return {"digits": digits.view(np.int64), "iteration": at, "good": good}
    if kind == "batch":
        r = m2.batch_run(held, iters=[case["iters"]] * len(held))
        return {"res64": r.res64.view(np.int64), "is_prime": r.is_prime}
    done = []
    with Server(8 << 30, case["quantum"]) as srv:
        for i, p in enumerate(held):
            srv.submit(i, p, m2.MODE_PRP, case["iters"])
        while len(done) < len(held):
            srv.step()
            done.extend(srv.poll())
    done.sort(key=lambda r: r.id)
    return {"res64": np.array([r.res64 for r in done], dtype=np.uint64).view(np.int64),
            "iters": np.array([r.iters for r in done]), "status": np.array([r.status for r in done]),
            "is_prime": np.array([r.is_prime for r in done])}


def _operations(p, fields="dual"):
    """Integer operations of one squaring: the 32 x 32 -> 64-bit products of a radix-4 transform, its inverse and the
    centre square (15 per product of two elements, 12 with one field), each a multiplication and an addition."""
    ln = _log2_digits(p, fields)
    h = 1 << (ln - 1)
    return 2 * (12 if fields == "gf61" else 15) * (0.75 * h * (ln - 1) + 2 * h)


def work(case):
    kind = case["kind"]
    if kind in ("advance", "gerbicz"):
        # the digits in and the digits out; under the check, the squarings of two blocks and of the verification, and
        # two for each of the three products
        fields = case.get("fields", "dual")
        k = case["iters"] if kind == "advance" else 3 * case["block"] + 6
        return {"bytes": 16 << _log2_digits(case["p"], fields), "flops": k * _operations(case["p"], fields)}
    # exponents in, residues and verdicts out; the operations of one draw of the exponents
    ps = _exponents(case, 0)
    return {"bytes": 17 * len(ps), "flops": sum(min(p, case["iters"]) * _operations(p) for p in ps)}


def _advance_exactly(x, p, mode, k):
    m = (1 << p) - 1
    for _ in range(k):
        x = x * x
        if mode == "ll":
            x -= 2
        elif mode == "prp3":
            x *= 3
        x = (x & m) + (x >> p)
        x = (x & m) + (x >> p)
        if x == m:
            x = 0
    return x


def exact(case, seed):
    if case["kind"] == "advance" and case["p"] * math.sqrt(case["p"]) * case["iters"] < 6e10:
        fields = case["fields"]
        p = case["p"]
        d = _digits(p, fields, seed)
        w = [int(v) for v in m2.layout(p, m2.FIELDS_GF61 if fields == "gf61" else m2.FIELDS_DUAL)[2]]
        x, at = 0, 0
        for v, wj in zip(d, w):
            x |= int(v) << at
            at += wj
        x = _advance_exactly(x % ((1 << p) - 1), p, case["mode"], case["iters"])
        out = np.zeros(len(w), dtype=np.int64)
        at = 0
        for j, wj in enumerate(w):
            out[j] = (x >> at) & ((1 << wj) - 1)
            at += wj
        return out
    if case["kind"] in ("batch", "serve"):
        ps = _exponents(case, seed)
        if sum(p ** 1.5 * min(p, case["iters"]) for p in ps) < 6e10:
            res = []
            for p in ps:
                x = _advance_exactly(3 % ((1 << p) - 1), p, "prp", min(p, case["iters"]))
                res.append(x & ((1 << 64) - 1))
            res = np.array(res, dtype=np.uint64).view(np.int64)
            return {"res64": res, "is_prime": None} if case["kind"] == "batch" else {"res64": res, "iters": None, "status": None, "is_prime": None}
    return None
