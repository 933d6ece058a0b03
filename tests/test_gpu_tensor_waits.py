"""The tensor walk when a wait runs out: one warp of each block stops before a
batch and waits, with a short limit, for a flag that nothing sets
(pps_debug_tensor_stall).  The kernels end by themselves, the call returns
PPS_ERR_TIMEOUT, and the same engine then gives the exact result."""
from __future__ import annotations

import time

import pytest

pytestmark = pytest.mark.gpu

CLOCKS = 2_000_000  # about 1 ms

# pmin, n values, kmax, sign: tiles of a unit 1, 3 and 4; 4- and 5-bit digits; both sides
SHAPES = [
    (42 * 10**12, 300_000, 9999, 1),
    (42 * 10**12, 600_000, 9999, 1),
    (42 * 10**12, 1_000_000, 9999, 2),
    ((1 << 62) - 10**9, 900_000, 9999, -1),
]


@pytest.fixture
def stall(pps):
    lib = pps.load()

    def set_stall(batch: int) -> None:
        assert lib.pps_debug_tensor_stall(batch, CLOCKS) == pps.PPS_OK

    yield set_stall
    lib.pps_debug_tensor_stall(-1, 0)


# before the first batch, before the third (both slots of the seeds' tables are
# then full) and before a later one, with work in flight
@pytest.mark.parametrize("batch", [0, 2, 3])
@pytest.mark.parametrize("pmin,span,kmax,sign", SHAPES)
def test_a_wait_that_runs_out(pps, stall, pmin, span, kmax, sign, batch):
    # 1,000 primes a block: some 30 batches
    jp = pps.normalize(pmin=pmin, pmax=pmin + 5 * 10**6, kmin=3, kmax=kmax, nmin=12_345, nmax=12_345 + span, sign=sign)
    with pps.Engine(0) as eng:
        eng.set_variant(32 if sign == pps.PPS_SIGN_TWIN else 31)
        want, st = eng.run_job(jp)
        stall(batch)
        with pytest.raises(pps.PPSError) as ei:
            eng.run_job(jp)
        assert ei.value.code == pps.PPS_ERR_TIMEOUT
        stall(-1)
        got, again = eng.run_job(jp)
        assert got.tobytes() == want.tobytes() and again.raw_hits == st.raw_hits and again.primes == st.primes


def test_one_wait_runs_out_not_one_a_part(pps):
    """A job of three parts: after the first part's time-out the other launches
    return at once, so the call takes one wait limit, not three."""
    clocks = 1_000_000_000  # about half a second
    jp = pps.normalize(pmin=42 * 10**12, pmax=42 * 10**12 + 75 * 10**6, kmin=1201, kmax=9999, nmin=2_000_000,
                       nmax=3_000_000)
    with pps.Engine(0) as eng:
        eng.set_variant(31)
        eng.run_job(jp)
        lib = pps.load()
        try:
            assert lib.pps_debug_tensor_stall(0, clocks) == pps.PPS_OK
            t0 = time.perf_counter()
            with pytest.raises(pps.PPSError) as ei:
                eng.run_job(jp)
            took = time.perf_counter() - t0
        finally:
            lib.pps_debug_tensor_stall(-1, 0)
        assert ei.value.code == pps.PPS_ERR_TIMEOUT and took < 1.0


def test_the_stall_needs_a_limit(pps):
    lib = pps.load()
    for clocks in (0, 1 << 40):
        assert lib.pps_debug_tensor_stall(0, clocks) == pps.PPS_ERR_INVALID_PARAM
