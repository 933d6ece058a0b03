"""The tensor walk on the GPU: its raw candidates are the oracle's, at the edges
of its tiles (112 columns, taken in pairs), units, digit sizes and batches."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P47, P62 = 1 << 47, 1 << 62

# pmin, how many primes, n values, kmax, sign
SHAPES = [
    (42 * 10**12, 1, 2_100, 9999, 1),           # the shortest n range it takes: 16 columns, one prime
    (42 * 10**12, 33, 300_000, 9999, 1),        # one whole tile; a batch of one unit after one of 32
    (10**12, 40, 111_111, 9999, -1),            # steps of 27, a ragged tile
    (10**13, 200, 1_000_000, 65_535, 1),        # a large k: many rows pass
    (42 * 10**12, 65, 600_000, 9999, 1),        # three tiles: a pair and a single one
    (42 * 10**12, 300, 1_000_000, 9999, -1),    # four tiles
    (P47 - 10**6, 40, 1_234_567, 9999, 1),      # the last p with 4-bit digits
    (P47 + 1, 40, 1_234_567, 9999, 1),          # the first with 5-bit digits
    (42 * 10**12, 20, 2_000_000, 9999, 1),      # two units to a prime
    (42 * 10**12, 10, 5_000_011, 9999, -1),     # eight
    (10**15, 40, 1_000_000, 999_999, 1),        # larger k, 5-bit digits
    (P62 - 10**6, 40, 900_000, 9999, -1),       # the largest p: steps above 32
    (42 * 10**12, 70, 1_000_000, 9999, 2),      # twin
    (10**12, 70, 250_000, 29_999, 2),           # twin, two sides' margins
]


def _raw(engine, jp, primes, variant):
    engine.set_variant(variant)
    try:
        return engine.check_primes_raw(jp, primes)
    finally:
        engine.set_variant(-1)


def _triples(raw):
    return sorted((int(h["p"]), int(h["k"]), int(h["n"])) for h in raw)


@pytest.mark.parametrize("pmin,np_,span,kmax,sign", SHAPES)
def test_tensor_walk_candidates(pps, engine, ora, pmin, np_, span, kmax, sign):
    nmin = 12_345
    spec = dict(pmin=pmin, pmax=min(pmin + 60 * np_ + 3000, P62), kmin=3, kmax=kmax, nmin=nmin, nmax=nmin + span,
                sign=sign)
    jp, op = pps.normalize(**spec), ora.normalize(**spec)
    primes = ora.sieve_range(jp.pmin, jp.pmax, jp.qmax)[:np_]
    variant = 32 if sign == pps.PPS_SIGN_TWIN else 31
    assert engine.check_primes(jp, primes[:1])[1].primes == 1
    engine.set_variant(variant)
    try:
        assert engine.check_primes(jp, primes)[1].variant == variant
    finally:
        engine.set_variant(-1)
    assert _triples(_raw(engine, jp, primes, variant)) == sorted(ora.raw_candidates(op, primes))


def test_tensor_walk_primes_outside_the_job(pps, engine, ora):
    """Its digits and margins are for [pmin, pmax): a list with other primes is
    walked all the same, by the recurrence."""
    spec = dict(pmin=42 * 10**12, pmax=42 * 10**12 + 10**4, kmin=3, kmax=9999, nmin=2000, nmax=602_000)
    jp = pps.normalize(**spec)
    primes = np.concatenate([ora.sieve_range(10**12, 10**12 + 3000, 0), ora.sieve_range(jp.pmin, jp.pmax, jp.qmax),
                             ora.sieve_range(10**15, 10**15 + 1000, 0)])
    assert _triples(_raw(engine, jp, primes, 31)) == _triples(_raw(engine, jp, primes, 0))


def test_tensor_walk_in_parts(pps, engine):
    """More primes than one launch's masks hold: the factors and candidates of
    the recurrence."""
    jp = pps.normalize(pmin=42 * 10**12, pmax=42 * 10**12 + (1 << 25) + (1 << 23), kmin=1201, kmax=9999,
                       nmin=2_000_000, nmax=3_000_000)
    got = []
    for variant in (31, 26):
        engine.set_variant(variant)
        try:
            fac, st = engine.run_job(jp)
        finally:
            engine.set_variant(-1)
        assert st.variant == variant
        got.append((st.raw_hits, fac.tobytes()))
    assert got[0] == got[1]


@pytest.mark.parametrize("segments", [0, 4])
def test_tensor_walk_in_a_batch(pps, segments):
    """Long and short n ranges, one-sided and twin, in one batch: the long ones
    leave the batch's walk kernel (with 4 segments to a wave, a part in each of
    several waves; the first wave holds nothing else), and every job's factors
    and counts are those of the recurrence alone."""
    specs = [
        dict(pmin=42 * 10**12, pmax=42 * 10**12 + 3 * 10**6, kmin=3, kmax=9999, nmin=2000, nmax=1_002_000, sign=1),
        dict(pmin=10**12, pmax=10**12 + 10**6, kmin=3, kmax=9999, nmin=2000, nmax=5000, sign=1),
        dict(pmin=10**12, pmax=10**12 + 2 * 10**6, kmin=3, kmax=9999, nmin=2000, nmax=602_000, sign=-1),
        dict(pmin=42 * 10**12, pmax=42 * 10**12 + 2 * 10**6, kmin=3, kmax=9999, nmin=2000, nmax=402_000, sign=2),
        dict(pmin=2 * 10**12, pmax=2 * 10**12 + 10**6, kmin=3, kmax=9999, nmin=3000, nmax=4000, sign=2),
        dict(pmin=P62 - 3 * 10**6, pmax=P62 - 10**6, kmin=3, kmax=9999, nmin=100_000, nmax=900_000, sign=-1),
    ]
    jobs = [pps.normalize(**s) for s in specs]
    with pps.Engine(0) as eng:
        if segments:
            eng.set_wave_segments(segments)
        per, st = eng.run_batch(jobs)
        count, total = eng.batch_job_primes(len(jobs))
        assert st.waves >= (2 if segments else 1)
    with pps.Engine(0) as eng:
        for i, jp in enumerate(jobs):
            # variant 22: twin jobs stay on the batched recurrence, alone
            eng.set_variant(22 if specs[i]["sign"] == pps.PPS_SIGN_TWIN else 0)
            want, one = eng.run_job(jp)
            assert per[i].tobytes() == want.tobytes(), specs[i]
            assert (int(count[i]), int(total[i])) == (int(one.primes), int(one.prime_sum))
