"""Moduli with a hit where one is wanted: odd p in [lo, hi) that divide
k 2^n + c for a chosen n.  p need not be prime (a walk's arithmetic needs p odd),
so it can be a product of small prime factors of one of the numbers k 2^n + c with
k in the range: the small primes that divide each are sieved for all k at once."""
from __future__ import annotations

import functools

import numpy as np

BOUND = 1 << 20


@functools.lru_cache(maxsize=1)
def _primes() -> np.ndarray:
    s = np.ones(BOUND, dtype=bool)
    s[:2] = False
    for i in range(2, 1025):
        if s[i]:
            s[i * i:: i] = False
    q = np.nonzero(s)[0].astype(np.uint64)
    return q[q > 2]


def _inv_pow2(n: int, q: np.ndarray) -> np.ndarray:
    """2^-n mod q for each q < 2^20."""
    r, b = np.ones_like(q), (q + np.uint64(1)) // np.uint64(2)
    while n:
        if n & 1:
            r = r * b % q
        b = b * b % q
        n >>= 1
    return r


def _subset(factors: list[int], lo: int, hi: int) -> int:
    """A product of some of the factors in [lo, hi), or 0."""
    seen = {1}
    for f in factors:
        seen |= {x * f for x in seen if x * f < hi}
        if len(seen) > 4096:
            break
    return next((x for x in sorted(seen) if lo <= x < hi), 0)


def plant(n: int, c: int, lo: int, hi: int, kmin: int, kmax: int, prefer: str = "high") -> tuple[int, int] | None:
    """(p, k): p in [lo, hi) divides k 2^n + c, k odd in [kmin, kmax] (the largest
    k or the smallest that gives one), or None."""
    k0 = kmin | 1
    count = (kmax - k0) // 2 + 1
    q = _primes()
    r = _inv_pow2(n, q)
    if c == 1:
        r = q - r
    # k0 + 2 j = r (mod q)
    j = (r + q - np.uint64(k0) % q) % q * ((q + np.uint64(1)) // np.uint64(2)) % q
    size = np.zeros(count)
    found: dict[int, list[int]] = {}
    for a, b in zip(j[q < count], q[q < count]):
        size[int(a):: int(b)] += np.log2(float(b))
    one = (q >= count) & (j < count)
    np.add.at(size, j[one].astype(np.int64), np.log2(q[one].astype(float)))
    ks = np.nonzero(size >= np.log2(float(lo)))[0]
    for jj in (ks[::-1] if prefer == "high" else ks):
        fs = [int(x) for x in q[j == np.uint64(jj) % q]]
        p = _subset(sorted(fs, reverse=True), lo, hi)
        if p:
            return p, k0 + 2 * int(jj)
    return None
