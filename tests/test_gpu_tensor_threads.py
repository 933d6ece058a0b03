"""Engines of several host threads on one GPU, each with tensor walks of another
plan: plans differ in the shared memory that they ask for, and no thread's call
may depend on another's."""
from __future__ import annotations

import threading

import pytest

pytestmark = pytest.mark.gpu

# pmin, n values, primes, calls: eight parts (their launches follow each other for a
# while), and calls of one part with less shared memory
JOBS = [(42 * 10**12, 1_000_000_000, 8192, 30), (42 * 10**12, 250_000, 64, 800), (42 * 10**12, 280_000, 64, 800),
        ((1 << 62) - 10**9, 600_000, 64, 800)]


def test_threads_with_different_plans(pps, ora):
    fails, done = [], []
    start = threading.Barrier(len(JOBS))

    def work(pmin, span, np_, calls):
        try:
            jp = pps.normalize(pmin=pmin, pmax=pmin + 50 * np_, kmin=3, kmax=9999, nmin=12_345, nmax=12_345 + span)
            primes = ora.sieve_range(jp.pmin, jp.pmax, jp.qmax)[:np_]
            with pps.Engine(0) as eng:
                eng.set_variant(31)
                want = eng.check_primes_raw(jp, primes).tobytes()
                start.wait(60)
                for _ in range(calls):
                    assert eng.check_primes_raw(jp, primes).tobytes() == want
            done.append(span)
        except BaseException as e:  # noqa: BLE001
            fails.append(e)
            start.abort()

    threads = [threading.Thread(target=work, args=j) for j in JOBS]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not fails and len(done) == len(JOBS), fails
