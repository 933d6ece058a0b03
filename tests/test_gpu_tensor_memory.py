"""The tensor walk when device memory is short (allocation failures injected on
the host): its masks shrink and the job is walked in more parts; with no room at
all the recurrence, which needs no masks, walks it.  The results do not change and
no call is refused."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPEC = dict(pmin=42 * 10**12, pmax=42 * 10**12 + 4 * 10**6, kmin=3, kmax=1 << 22, nmin=12_345, nmax=1_012_345)
TWIN = dict(SPEC, sign=2)


@pytest.fixture
def fail(pps):
    lib = pps.load()
    yield lib.pps_debug_fail_allocs
    lib.pps_debug_fail_allocs(0, 0)


def _warm(pps, eng, jp, primes):
    """Every buffer but the masks: the calls that follow, by the recurrence."""
    eng.set_split(1)
    eng.run_job(pps.normalize(**SPEC))
    eng.run_job(jp)
    eng.check_primes_raw(jp, primes)
    eng.run_batch([jp])
    eng.set_split(0)


def _run_job(eng, jp, primes, want, tensor):
    fac, st = eng.run_job(jp)
    assert fac.tobytes() == want["fac"] and st.raw_hits == want["raw_hits"] and (st.variant in (31, 32)) == tensor


def _check_primes(eng, jp, primes, want, tensor):
    fac, st = eng.check_primes(jp, primes)
    assert fac.tobytes() == want["fac"] and (st.variant in (31, 32)) == tensor


def _check_primes_raw(eng, jp, primes, want, tensor):
    assert eng.check_primes_raw(jp, primes).tobytes() == want["raw"]


def _run_batch(eng, jp, primes, want, tensor):
    per, st = eng.run_batch([jp])
    assert per[0].tobytes() == want["fac"] and st.raw_hits == want["raw_hits"]


# one failure: masks of a quarter; two: a sixteenth, or the least; many: none at all
@pytest.mark.parametrize("count,tensor", [(1, True), (2, True), (100, False)])
@pytest.mark.parametrize("spec", [SPEC, TWIN])
@pytest.mark.parametrize("call", [_run_job, _check_primes, _check_primes_raw, _run_batch])
def test_no_room_for_the_masks(pps, engine, fail, call, spec, count, tensor):
    jp = pps.normalize(**spec)
    primes = engine.sieve_range(jp.pmin, jp.pmax, want_primes=True, cap=1 << 20)[0]
    fac, st = engine.run_job(jp)
    assert st.variant in (31, 32) and len(fac)
    want = dict(fac=fac.tobytes(), raw_hits=st.raw_hits, raw=engine.check_primes_raw(jp, primes).tobytes())
    with pps.Engine(0) as eng:
        _warm(pps, eng, jp, primes)
        fail(0, count)
        if call is _run_batch and count == 1:
            fail(1, 1)  # (a batch makes room for a few primes first, then for a wave's)
        call(eng, jp, primes, want, tensor)
        assert fail(0, 0) >= 1
        call(eng, jp, primes, want, True)


@pytest.mark.parametrize("count", [1, 100])
def test_no_room_for_the_copy_of_a_pinned_list(pps, engine, fail, count):
    """A page-locked list is walked where it is; `count` 100: nor is there room for the masks."""
    import torch

    jp = pps.normalize(**SPEC)
    primes = engine.sieve_range(jp.pmin, jp.pmax, want_primes=True, cap=1 << 20)[0]
    raw = engine.check_primes_raw(jp, primes).tobytes()
    host = torch.from_numpy(primes.view(np.int64)).pin_memory().numpy().view(np.uint64)
    with pps.Engine(0) as eng:
        eng.check_primes_raw(jp, host[:10])  # the candidate buffers, and masks for ten
        fail(1 if count == 1 else 0, count)  # (the masks' come first)
        assert eng.check_primes_raw(jp, host).tobytes() == raw
        assert fail(0, 0) >= 1
