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
