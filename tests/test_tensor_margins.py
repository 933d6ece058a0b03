"""The tensor walk's screening never drops a hit: the largest errors of the
tested fraction, from a numpy model of the operand rows and of the accumulator,
against the margins of the plans that the library makes (CPU only).

All errors are in 2^-16, the unit of the tested fraction.  A row value A, in
units of 2^-12, enters as a whole number h and the rest l in fp16; a prime's sum
has 15 slots with balanced digits up to half the base.  The sum of the l products
is cut towards zero to a quarter of the accumulator's last bit (1; base 32: 2),
the whole, which is positive, to its last bit.  In base 32 the test doubles two
fractions of a register at once, and the lower one's top bit moves into the upper
one's last place."""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import pytest

BASES = {4: 16, 5: 32}


class Plan(ctypes.Structure):
    _fields_ = [(n, ctypes.c_uint32) for n in ("s", "nb", "units", "digits", "pitch", "off", "thr")] + [
        ("cost", ctypes.c_double)]


@pytest.fixture(scope="module")
def plan(pps):
    lib = pps.load()
    fn = getattr(lib, "_ZN3pps11tensor_planEPK14pps_job_paramsPNS_10TensorPlanE")
    fn.restype = ctypes.c_bool

    def of(jp):
        p = Plan()
        return p if fn(ctypes.byref(jp), ctypes.byref(p)) else None

    return of


def _slot(x: np.ndarray):
    """split_pair and half2_of for signed 32-bit row values: h and l, in 2^-12."""
    w = x.astype(np.float32).astype(np.float64)  # int to float, to nearest
    magic = 12582912.0
    h = (w / 2**20 + magic).astype(np.float32).astype(np.float64) - magic
    l = (w / 2**20 - h).astype(np.float32).astype(np.float16).astype(np.float64)
    return h, l


def _worst_slot():
    rng = np.random.default_rng(3)
    x = rng.integers(-(2**31), 2**31, size=4_000_000).astype(np.int32)
    h, l = _slot(x)
    err = (h + l - x / 2**20) * 16.0  # 2^-12 to 2^-16
    assert abs(h).max() <= 2048 and abs(l).max() <= 0.5  # h: exact in fp16
    return x, err


def _bounds(digits: int):
    """How far the tested fraction may lie below and above the true one, without v_b's tail."""
    half = BASES[digits] // 2
    row = 15 * half * (3 * 2.0**-14 * 16 + 2.0**-16)  # l's two roundings; the bits of K_a beyond 32
    last = half / 8
    return row + last, row + last / 4 + (1.0 if digits == 5 else 0.0)


def test_row_values_err_by_three_2e_minus_14():
    _, err = _worst_slot()
    assert 2.9 * 2.0**-10 < abs(err).max() <= 3 * 2.0**-10


@pytest.mark.parametrize("digits", [4, 5])
def test_sums_at_their_worst_stay_within_the_bounds(digits):
    """Sums of the rows and digits whose errors add up, through the accumulator:
    the bounds hold, and the errors come near them."""
    half, rng = BASES[digits] // 2, random.Random(digits)
    x, err = _worst_slot()
    worst = x[np.argsort(-abs(err))[:4000]]
    last = half / 8
    below, above = _bounds(digits)
    lo = hi = 0.0
    for trial in range(4000):
        want = 1 if trial & 1 else -1  # the sign the errors add up to
        v = np.array([worst[rng.randrange(len(worst))] for _ in range(15)])
        h, l = _slot(v)
        e = (h + l - v / 2**20) * 16.0
        d = np.where(e * want > 0, half - 1, -half) if trial % 3 else np.where(e > 0, want, -want) * rng.randint(1, half - 1)
        lsum = float((d * l).sum()) * 16.0
        cut = math.copysign(math.floor(abs(lsum) * 4 / last) / 4 * last, lsum)
        got = math.floor((float((d * h).sum()) * 16.0 + cut) / last) * last  # h products: whole multiples of 16
        true = float((d * v.astype(np.float64)).sum()) / 2**20 * 16.0
        lo, hi = min(lo, got - true), max(hi, got - true)
    carry = 1.0 if digits == 5 else 0.0
    assert -below <= lo and hi + carry <= above
    assert hi + carry > above - last / 2 - 0.2


@pytest.mark.parametrize("sign", [1, -1, 2])
@pytest.mark.parametrize("digits", [4, 5])
def test_plans_leave_room_for_the_worst_errors(pps, plan, digits, sign):
    rng = random.Random(10 * digits + sign)
    below, above = _bounds(digits)
    seen = 0
    for _ in range(600):
        lo, hi = (36.0, 46.9) if digits == 4 else (47.1, 61.9)
        pmin = int(2.0 ** rng.uniform(lo, hi))
        kmax = int(2.0 ** rng.uniform(8, min(36, math.log2(pmin) - 12)))
        span, nmin = int(2.0 ** rng.uniform(11, 27)), rng.randrange(200, 10**6)
        try:
            jp = pps.normalize(pmin=pmin, pmax=pmin + rng.randrange(10**4, pmin // 8), kmin=3, kmax=kmax, nmin=nmin,
                               nmax=nmin + span, sign=sign)
        except pps.PPSError:
            continue
        t = plan(jp)
        if t is None or t.digits != digits:
            continue
        seen += 1
        tail = math.ldexp(jp.pmax, 16 - (62 if digits == 4 else 77))
        eps = jp.kmax / jp.pmin * 65536.0 * 2.0 ** (t.s - 1)
        # the smallest hit (twin: the other side's, at -eps) stays above zero, the largest passes
        assert t.off - (eps if sign == 2 else 0.0) - tail - below >= 0.0
        assert math.floor(t.off + eps + tail + above) < t.thr, (jp.pmin, jp.kmax, t.s, eps, tail)
    assert seen > 100
