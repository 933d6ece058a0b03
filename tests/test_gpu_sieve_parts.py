"""The device sieve of a batch of more than 3,072 segments (2^18 odd candidates
each), which goes in parts: count and sum of its primes against the CPU oracle."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

SEG = 1 << 19  # p width of a segment


@pytest.mark.parametrize("width", [3072 * SEG, 3072 * SEG + 2, 4095 * SEG + 1000])
def test_sieve_in_parts_matches_oracle(pps, engine, ora, width):
    lo, qmax = 3 * 10**11 + 1, 600_000  # every prime up to the root
    _, count, total = engine.sieve_range(lo, lo + width, qmax)
    want = ora.fingerprint(lo, lo + width, qmax)
    assert (int(count), int(total)) == (int(want[0]), int(want[1]))
