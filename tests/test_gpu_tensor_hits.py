"""The tensor walk finds every hit: lists of moduli with a hit planted at the
edges of its units, tiles, rows and steps, for both digit sizes, and lists and
batches with many natural hits.  Every list of candidates is the oracle's (or the
recurrence's), and none is empty."""
from __future__ import annotations

import ctypes
import random

import numpy as np
import pytest

from planted import plant
from test_tensor_margins import Plan

P47, P62 = 1 << 47, 1 << 62


def _plan(pps, jp) -> Plan:
    fn = getattr(pps.load(), "_ZN3pps11tensor_planEPK14pps_job_paramsPNS_10TensorPlanE")
    fn.restype = ctypes.c_bool
    p = Plan()
    assert fn(ctypes.byref(jp), ctypes.byref(p))
    return p


def _triples(raw):
    return sorted((int(h["p"]), int(h["k"]), int(h["n"])) for h in raw)


def _walk(engine, jp, primes, variant):
    engine.set_variant(variant)
    try:
        assert engine.check_primes(jp, primes)[1].variant == variant
        return engine.check_primes_raw(jp, primes)
    finally:
        engine.set_variant(-1)


def _planted(pps, ora, spec, seed, count=40):
    """Moduli with a hit at the edges of the job's plan and at random places, and
    the hits (p, k, n)."""
    jp = pps.normalize(**spec)
    t, rng = _plan(pps, jp), random.Random(seed)
    ks = (jp.kmin, jp.kmax)
    cols = [b for b in (0, 1, 31, 32, 63, 64, 95, 96, 111, 112, 223, 224, 335, 336) if b < t.nb] + [t.nb - 1]
    want = []

    def put(n, prefer):
        if not jp.nmin <= n < jp.nmax:
            return
        c = rng.choice((1, -1)) if jp.sign == pps.PPS_SIGN_TWIN else jp.sign
        r = plant(n, c, jp.pmin, jp.pmax, *ks, prefer)
        if r:
            want.append((r[0], r[1], n))

    at = lambda unit, row, b, i: jp.nmin + t.s * ((unit * 128 + row) * t.nb + b) + i
    for unit in sorted({0, t.units // 2, t.units - 1}):
        for row in (0, 31, 32, 127):
            for b in cols:
                # the largest fraction that a hit can have (i = s - 1, the largest k) and the smallest
                put(at(unit, row, b, t.s - 1), "high")
                put(at(unit, row, b, 0), "low")
    put(jp.nmin, "low")
    put(jp.nmax - 1, "high")
    for _ in range(count):
        put(rng.randrange(jp.nmin, jp.nmax), rng.choice(("high", "low")))
    return jp, want


# pmin, pmax, n values, sign; steps of up to 18 n, of 12 and of 34 (above 32, in two)
PLANTED = [
    (42 * 10**12, 44 * 10**12, 300_000, 1),      # a tile
    (42 * 10**12, 44 * 10**12, 1_000_000, -1),   # four tiles
    (10**12, 105 * 10**10, 150_000, 1),
    (P47 - (1 << 42), P47, 700_000, 1),          # the largest p with 4-bit digits
    (P47 + 1, P47 + (1 << 42), 300_000, 1),      # the smallest with 5-bit digits
    (P47 + 1, P47 + (1 << 42), 1_000_000, -1),
    (10**15, 105 * 10**13, 1_000_000, 1),
    (P62 - (1 << 57), P62, 300_000, -1),         # the largest p
    (P62 - (1 << 57), P62, 900_000, -1),
    (P62 - (1 << 57), P62, 900_000, 1),
    (42 * 10**12, 44 * 10**12, 1_000_000, 2),    # both sides
    (1 << 50, 17 << 46, 700_000, 2),
    (42 * 10**12, 44 * 10**12, 5_000_011, 1),    # several units to a modulus
    (P62 - (1 << 57), P62, 12_000_000, -1),
]


@pytest.mark.gpu
@pytest.mark.parametrize("pmin,pmax,span,sign", PLANTED)
def test_planted_hits(pps, engine, ora, pmin, pmax, span, sign):
    spec = dict(pmin=pmin, pmax=pmax, kmin=3, kmax=9999, nmin=12_345, nmax=12_345 + span, sign=sign)
    jp, want = _planted(pps, ora, spec, seed=span + sign)
    assert len(want) > 60
    primes = np.array([w[0] for w in want], dtype=np.uint64)
    raw = _walk(engine, jp, primes, 32 if sign == pps.PPS_SIGN_TWIN else 31)
    assert all(int(primes[int(h["idx"]) & 0x7fffffff]) == int(h["p"]) for h in raw)
    got = _triples(raw)
    assert set(want) <= set(got)
    assert got == sorted(ora.raw_candidates(ora.normalize(**spec), primes))


def test_planted_hits_are_the_oracles(pps, ora):
    """The lists themselves, without a GPU: the oracle finds each planted hit."""
    for pmin, pmax, span, sign in PLANTED[::4]:
        spec = dict(pmin=pmin, pmax=pmax, kmin=3, kmax=9999, nmin=12_345, nmax=12_345 + span, sign=sign)
        _, want = _planted(pps, ora, spec, seed=span + sign, count=5)
        want = want[::7]
        primes = np.array([w[0] for w in want], dtype=np.uint64)
        assert want and set(want) <= set(ora.raw_candidates(ora.normalize(**spec), primes))


# pmin, how many primes, n values, kmax, sign, the least number of hits
NATURAL = [
    (10**12, 1500, 600_000, 50_001, 1, 10),
    (42 * 10**12, 40, 1_000_000, 1 << 26, -1, 20),
    (P47 + 1, 40, 1_000_000, 1 << 29, 1, 40),
    (10**15, 40, 1_000_000, 1 << 34, -1, 150),      # several to a prime,
    (P62 - 10**9, 2000, 900_000, 1 << 37, -1, 15),
    (P62 - 10**9, 2000, 900_000, 1 << 37, 1, 15),
    (1 << 50, 60, 600_000, 1 << 30, 2, 20),
]


@pytest.mark.gpu
@pytest.mark.parametrize("pmin,np_,span,kmax,sign,least", NATURAL)
def test_natural_hits(pps, engine, ora, pmin, np_, span, kmax, sign, least):
    nmin = 54_321
    spec = dict(pmin=pmin, pmax=min(pmin + 60 * np_ + 3000, P62), kmin=3, kmax=kmax, nmin=nmin, nmax=nmin + span,
                sign=sign)
    jp = pps.normalize(**spec)
    primes = ora.sieve_range(jp.pmin, jp.pmax, jp.qmax)[:np_]
    got = _triples(_walk(engine, jp, primes, 32 if sign == pps.PPS_SIGN_TWIN else 31))
    assert len(got) >= least
    assert got == sorted(ora.raw_candidates(ora.normalize(**spec), primes))


@pytest.mark.gpu
@pytest.mark.parametrize("pinned", [False, True])
def test_lists_with_primes_outside_the_job(pps, engine, ora, pinned):
    """A prime outside [pmin, pmax) anywhere in the list: the whole list's
    candidates, hits of the outside ones among them."""
    import torch

    spec = dict(pmin=42 * 10**12, pmax=44 * 10**12, kmin=3, kmax=9999, nmin=12_345, nmax=612_345)
    jp, want = _planted(pps, ora, spec, seed=5)
    far = [dict(spec, pmin=45 * 10**12, pmax=47 * 10**12), dict(spec, pmin=10**15, pmax=102 * 10**13)]
    out = [w for f, s in zip(far, (6, 7)) for w in _planted(pps, ora, f, seed=s)[1][:20]]
    for where in (0, len(want) // 2, len(want)):
        both = want[:where] + out + want[where:]
        primes = np.array([w[0] for w in both], dtype=np.uint64)
        if pinned:
            host = torch.from_numpy(primes.view(np.int64)).pin_memory()
            primes = host.numpy().view(np.uint64)
        got = _triples(engine.check_primes_raw(jp, primes))
        assert set(both) <= set(got)
        assert got == sorted(ora.raw_candidates(ora.normalize(**spec), primes))


@pytest.mark.gpu
def test_batch_jobs_with_hits_leave_for_the_tensor_walk(pps):
    """Long n ranges of a batch with many candidates: they are walked by launches
    of their own (two more a job than with the recurrence alone), and factors,
    counts and sums are the recurrence's."""
    specs = [
        dict(pmin=42 * 10**12, pmax=42 * 10**12 + 2 * 10**6, kmin=3, kmax=1 << 24, nmin=2000, nmax=1_002_000, sign=1),
        dict(pmin=P47 + 1, pmax=P47 + 2 * 10**6, kmin=3, kmax=1 << 28, nmin=2000, nmax=1_002_000, sign=-1),
        dict(pmin=P62 - 10**9, pmax=P62 - 10**9 + 2 * 10**6, kmin=3, kmax=1 << 37, nmin=20_000, nmax=920_000, sign=-1),
        dict(pmin=1 << 50, pmax=(1 << 50) + 2 * 10**6, kmin=3, kmax=1 << 30, nmin=3000, nmax=803_000, sign=2),
        dict(pmin=10**12, pmax=10**12 + 10**6, kmin=3, kmax=9999, nmin=2000, nmax=5000, sign=1),
    ]
    jobs = [pps.normalize(**s) for s in specs]
    runs = []
    for variant in (-1, 0):
        with pps.Engine(0) as eng:
            if variant == 0:
                eng.set_split(1)  # parts of the recurrence: no job leaves, twin ones included
            eng.run_batch(jobs)
            before = eng.launches
            per, st = eng.run_batch(jobs)
            runs.append((eng.launches - before, st.waves, [f.tobytes() for f in per], st.raw_hits,
                         [c.tolist() for c in eng.batch_job_primes(len(jobs))]))
    (launches, waves, *got), (alone, waves0, *want) = runs
    assert waves == waves0 == 1 and launches == alone + 2 * 4
    assert got == want and all(len(f) for f in got[0][:4])


@pytest.mark.gpu
@pytest.mark.parametrize("where", [0, -1])
def test_a_list_with_one_prime_outside_is_walked_once(pps, engine, where):
    """One prime outside the job's range, first or last of 300,000: the call takes
    what the recurrence alone takes, not that and a tensor walk."""
    import time

    spec = dict(pmin=42 * 10**12, pmax=42 * 10**12 + 10**7, kmin=3, kmax=9999, nmin=12_345, nmax=1_012_345)
    jp = pps.normalize(**spec)
    primes = engine.sieve_range(jp.pmin, jp.pmax, want_primes=True, cap=400_000)[0][:300_000].copy()
    assert engine.check_primes(jp, primes)[1].variant == 31
    primes[where] = 45 * 10**12 + 1

    def best():
        took = []
        for _ in range(9):
            t0 = time.perf_counter()
            _, st = engine.check_primes(jp, primes)
            took.append(time.perf_counter() - t0)
        return min(took), st.variant

    once, variant = best()
    assert variant != 31
    engine.set_variant(variant)
    try:
        alone, _ = best()
    finally:
        engine.set_variant(-1)
    assert once < 1.2 * alone, (once, alone)
