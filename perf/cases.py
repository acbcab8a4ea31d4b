"""The work this framework is asked to do, as timed cases.

A case names a kind of call and its sizes; a pass goes through the public entry points only: the
kite API (kite_square_n, kite_mul, kite_get_limbs, kite_prp, kite_llr), the batched engine
(kc_batch_*) and groups of the integer-NTT engine (kn_groups_square).  Every output is a whole
number modulo N = k*2^n-1 (little-endian 64-bit limbs) or a verdict, so a pass is right only if
every bit is.

  block      one Gerbicz block of one test: `squarings` squarings of x, then d <- d*x, and the two
             numbers read back (what a checkpoint writes).  squarings = 1 without the product is
             the smallest call: square once and look at the result.
  prp, llr   a whole test of a small number through kite_prp / kite_llr: context, start, blocks,
             checks, tail, verdict.
  batch      one Gerbicz block of many Fermat tests advanced together (kc_batch_step), the
             numbers read back.
  served     the same for a request loop's mix: Fermat and LLR tests of very different lengths in
             one batch; a test that finishes is replaced, as the loop admits the next request.
  ntt_group  many tests on the integer-NTT engine, two groups on two streams.
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np

from ahnum_gb300 import kite, native
from ahnum_gb300.ntt_group import NttGroup
from ahnum_gb300.tune import load_gb300_tuning

SMALL_PRIMES = [p for p in range(3, 1000, 2) if all(p % q for q in range(3, int(p ** 0.5) + 1, 2))]


def listed():
    return [
        # one squaring and a look at the residue: what a call costs at the smallest size in use
        {"name": "one_squaring_n20000", "kind": "block", "backend": "cuda", "k": 9357, "n": 20000, "squarings": 1, "product": False},
        # a small test alone, at kite_prp's default block (the square root of n)
        {"name": "block_n20000", "kind": "block", "backend": "cuda", "k": 9357, "n": 20000, "squarings": 141, "product": True},
        # the two sizes of a test run alone that the benchmark names: FFT lengths 28672 and 49152
        {"name": "block_n369717", "kind": "block", "backend": "cuda", "k": 9357, "n": 369717, "squarings": 608, "product": True},
        {"name": "block_n662695", "kind": "block", "backend": "cuda", "k": 9001, "n": 662695, "squarings": 814, "product": True},
        # the large single test: a megaword transform, part of a block
        {"name": "block_n24715281", "kind": "block", "backend": "cuda", "k": 187, "n": 24715281, "squarings": 200, "product": True},
        # whole tests of small numbers, from the call to the verdict
        {"name": "prp_n12000", "kind": "prp", "n": 12000},
        {"name": "llr_n8000", "kind": "llr", "n": 8000},
        # the benchmark's batch: mixed FFT lengths 20480-51200, a block of 1000 squarings
        {"name": "batch_256", "kind": "batch", "tests": 256, "lo": 300000, "hi": 700000, "block": 1000},
        # the request loop's mix, four Fermat tests to one LLR test, n over more than a decade
        {"name": "served_16", "kind": "served", "tests": 16, "lo": 100000, "hi": 4000000, "block": 200},
        # the exact integer engine, alone and in groups
        {"name": "ntt_block_n369717", "kind": "block", "backend": "ntt", "k": 9357, "n": 369717, "squarings": 608, "product": True},
        {"name": "ntt_group_128", "kind": "ntt_group", "tests": 128, "lo": 300000, "hi": 700000, "squarings": 64},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: sizes log-uniform, n and k odd and even, smooth or not."""
    kind = rng.choice(["block", "block", "block", "prp", "llr", "batch", "batch", "served", "ntt", "ntt_group"])
    if kind in ("block", "ntt"):
        n = _log_uniform(rng, 2048, 25000000 if kind == "block" else 10000000)
        k = _log_uniform(rng, 3, 9999) | 1
        most = min(2000, max(32, math.isqrt(n)), max(20, 200 * 25000000 // n))
        squarings = _log_uniform(rng, 1, most)
        return {"kind": "block", "backend": "cuda" if kind == "block" else "ntt", "k": k, "n": n,
                "squarings": squarings, "product": squarings > 1}
    if kind in ("prp", "llr"):
        return {"kind": kind, "n": _log_uniform(rng, 2500, 16000)}
    if kind == "batch":
        return {"kind": "batch", "tests": _log_uniform(rng, 2, 192), "lo": 300000, "hi": 700000, "block": rng.randrange(100, 1001)}
    if kind == "served":
        return {"kind": "served", "tests": rng.randrange(2, 25), "lo": 100000, "hi": 4000000, "block": rng.randrange(50, 301)}
    return {"kind": "ntt_group", "tests": _log_uniform(rng, 2, 192), "lo": 300000, "hi": 700000, "squarings": rng.randrange(8, 129)}


# ---- sizes ------------------------------------------------------------------------------------


def _sizes(case):
    """n of each of the case's tests: the same for every seed."""
    rng = random.Random(case["tests"])
    out = []
    for _ in range(case["tests"]):
        if case["kind"] == "served":
            out.append(_log_uniform(rng, case["lo"], case["hi"]))
        else:
            out.append(rng.randrange(case["lo"], case["hi"] + 1))
    return out


def _length(n, k):
    """Words of the shortest real transform for N at the reference model's bits per word."""
    L = 64.0
    for _ in range(40):
        L = n / (21.24 - 0.305 * (math.log2(L) - 12) - 0.5 * math.log2(k))
    return L


def work(case):
    """Bytes: every number read once and written once.  Operations: 5 L log2(L/2) + 24 L for each
    squaring or product of an L-word number (forward and inverse real transform, pointwise
    square, weights, rounding and carries)."""
    def flops(n, k):
        L = _length(n, k)
        return 5 * L * math.log2(L / 2) + 24 * L

    if case["kind"] == "block":
        numbers = 2 if case["product"] else 1
        return {"bytes": numbers * 2 * case["n"] / 8,
                "flops": (case["squarings"] + (numbers - 1)) * flops(case["n"], case["k"])}
    if case["kind"] in ("prp", "llr"):
        return {"bytes": 2 * case["n"] / 8, "flops": case["n"] * flops(case["n"], 9999)}
    per = case["block"] + 1 if "block" in case else case["squarings"]
    sizes = _sizes(case)
    return {"bytes": sum(2 * n / 8 for n in sizes), "flops": per * sum(flops(n, 5000) for n in sizes)}


# ---- inputs -----------------------------------------------------------------------------------


def _candidate(rng, n):
    """k odd in [3, 9999] with no prime factor of k*2^n-1 below 1000: what a sieve leaves."""
    powers = [(p, pow(2, n, p)) for p in SMALL_PRIMES]
    while True:
        k = rng.randrange(3, 10000, 2)
        if all((k * t - 1) % p for p, t in powers):
            return k


class _State:
    def __init__(self, case):
        self.case = case
        self.lib = native.load()
        load_gb300_tuning(self.lib)
        self.owner = None  # what holds the device memory

    def __del__(self):
        if self.owner is not None:
            self.owner.close()


def prepare(case, seed):
    s = _State(case)
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "block":
        s.owner = kite.Ctx(case["k"], case["n"], backend=kite.CUDA if case["backend"] == "cuda" else kite.CUDA_NTT)
        bits = case["n"] - 1
        s.x = s.owner.num(rng.getrandbits(bits))
        s.d = s.owner.num(rng.getrandbits(bits))
    elif kind in ("prp", "llr"):
        s.k = _candidate(rng, case["n"])
    elif kind in ("batch", "served"):
        s.owner = kite.Batch(gerbicz_block=case["block"])
        s.lib.kc_batch_stagger_checks(s.owner.h, 1)
        s.tests = []
        for i, n in enumerate(_sizes(case)):
            k = _candidate(rng, n)
            s.tests.append((k, n, kind == "served" and i % 5 == 4))
        s.slots = [_admit(s, t) for t in s.tests]
    else:
        s.tests = [(rng.randrange(3, 10000, 2), n) for n in _sizes(case)]
        s.owner = NttGroup(s.tests)
        # full-size residues, as in the middle of a test
        for (k, n), e, x in zip(s.tests, s.owner.engines, s.owner.nums):
            limbs = (C.c_uint64 * s.lib.kn_limbs(e))()
            v = rng.getrandbits(n - 1)
            C.memmove(limbs, v.to_bytes(8 * len(limbs), "little"), 8 * len(limbs))
            if s.lib.kn_set_limbs(e, x, limbs) != 0:
                raise RuntimeError("kn_set_limbs failed")
    return s


def _admit(s, test):
    k, n, llr = test
    slot = s.owner.add_llr(k, n) if llr else s.owner.add_fermat(k, n)
    if slot < 0:
        raise RuntimeError(f"{k}*2^{n}-1 was not admitted")
    return slot


# ---- a pass -----------------------------------------------------------------------------------


def _limbs(count):
    a = np.empty(count, np.uint64)
    return a, a.ctypes.data_as(native.u64p)


def run(s):
    kind, case = s.case["kind"], s.case
    if kind == "block":
        c = s.owner
        c.square(s.x, case["squarings"])
        if case["product"]:
            c.mul(s.d, s.x)
        out = []
        for num in (s.x, s.d) if case["product"] else (s.x,):
            a, p = _limbs(c.nlimbs)
            c.lib.kite_get_limbs(c.h, num.h, p)
            out.append(a)
        c.check()
        return out
    if kind == "prp":
        r = kite.prp(s.k, case["n"])
        return [r.rc, np.uint64(r.res64), r.is_prp, r.gerbicz_errors]
    if kind == "llr":
        r = kite.llr(s.k, case["n"])
        return [r.rc, np.uint64(r.res64), r.is_prime, np.uint64(r.factor), r.P]
    if kind in ("batch", "served"):
        b = s.owner
        b.step(1)
        out = []
        for i, (slot, test) in enumerate(zip(s.slots, s.tests)):
            a, p = _limbs((test[1] + 127) // 64)
            if s.lib.kc_batch_read(b.h, slot, p) != 0:
                raise RuntimeError("kc_batch_read failed")
            out.append(a)
            if b.result(slot)[0]:  # finished: the next request takes its place
                b.release(slot)
                s.slots[i] = _admit(s, test)
        return np.concatenate(out)
    s.owner.square(case["squarings"])
    out = []
    for e, x in zip(s.owner.engines, s.owner.nums):
        a, p = _limbs(s.lib.kn_limbs(e))
        if s.lib.kn_get_limbs(e, x, p) != 0:
            raise RuntimeError("kn_get_limbs failed")
        out.append(a)
    return np.concatenate(out)


def exact(case, seed):
    """Every output is a whole number: there is nothing to round."""
    return None
