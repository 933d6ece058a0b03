"""Every wait of the tensor walk's kernels has a limit: read from the sources, no
GPU.  A wait without one could outlast a role that left after a time-out, and
the block would never end."""
from __future__ import annotations

import re

from conftest import PKG

FILES = ("pps_tensor.cu", "pps_tcgen05.cuh")


def _code(name: str) -> str:
    src = (PKG / "csrc" / name).read_text()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", src, flags=re.S))


def test_no_named_barriers():
    """A named barrier joins some of a block's warps without a limit; the only
    barriers are the block's own, which every role reaches when its loops end."""
    for name in FILES:
        assert not re.search(r"\b(bar|barrier)\.(cta\.)?(sync|red|arrive)\b|__named_barrier|\bbarrier_sync", _code(name)), name


def test_every_mbarrier_wait_goes_through_the_bounded_one():
    tc, tw = _code("pps_tcgen05.cuh"), _code("pps_tensor.cu")
    assert tc.count("mbarrier.try_wait") + tc.count("mbarrier.test_wait") == 1
    assert "mbarrier." not in tw.replace("mbarrier_init.release", "")
    body = tc[tc.index("bool mbar_wait("):]
    body = body[: body.index("\n}\n")]
    assert tc.count("mbar_try_wait(") == 1 + body.count("mbar_try_wait(") and "mbar_try_wait(" not in tw
    assert "limit" in body.lower() and "return false" in body


def _block_end(units, npairs, stages, waits):
    """The commits' arrivals on the operand stages that may still be under way
    when a block of `units` units ends.  Each unit's pairs of tiles go to the two
    MMA warps in turn; a warp with a pair of the unit commits to its stage, one
    without arrives plainly.  `waits(unit_no)`: the units whose stages both warps
    wait for at the end."""
    skip, commits = [0, 1], set()
    for u in range(units):
        for h in range(2):
            if skip[h] < npairs:
                commits.add((u % stages, u // stages))
                while skip[h] < npairs:
                    skip[h] += 2
            skip[h] -= npairs
    # a build group refills a stage, and so waits for its use before, while units come
    seen = {(u % stages, u // stages - 1) for u in range(units) if u >= stages}
    seen |= {(u % stages, u // stages) for u in waits(units)}
    return commits - seen


def test_no_arrival_outlasts_the_block():
    """Waiting for the last unit's stage alone leaves the other half's last commit
    under way where a unit has one pair of tiles; each stage's last use does not."""
    src = _code("pps_tensor.cu")
    stages = int(re.search(r"TW_STAGES = (\d+)", src).group(1))
    last = lambda n: [n - 1] if n else []
    each = lambda n: [n - i for i in range(1, min(stages, n) + 1)]
    assert _block_end(7, 1, stages, last)
    for npairs in (1, 2, 3):
        for units in range(40):
            assert not _block_end(units, npairs, stages, each), (npairs, units)
    # and the kernel does that, and drains its MMAs whether or not a wait ran out
    end = src[src.index("free_par ^= 1u"):]
    assert re.search(r"i <= min\(TW_STAGES, unit_no\); \+\+i\)\s*ok = mbar_wait<0>\(abe0 \+ \(unit_no - i\) % TW_STAGES", end)
    assert end.index("mma_commit(smem_addr(&sh->drain[half]))") < end.index("tmem_dealloc")
