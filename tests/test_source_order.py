"""Orderings that no run can be relied on to show: read from the kernels' sources."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "flashrnn_b200" / "csrc"


def _body(text: str, start: str) -> str:
    """The braces that follow ``start``."""
    at = text.index("{", text.index(start))
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i + 1]
    raise AssertionError(start)


def test_scratch_in_a_tma_ring_is_fenced_before_tma_writes_it():
    """Fragments pass through the ring that TMA fills afterwards: the last ordinary access of the scratch is followed by a proxy
    fence, and that by the barrier behind which the I/O warp asks for the first tiles."""
    load = _body((CSRC / "recurrent_reg.cuh").read_text(), "void reg_load_rows(")
    through_scratch = load[:load.index("} else {")]
    assert through_scratch.rindex("ldsm_x4(scratch") < through_scratch.rindex("fence_proxy_async_smem();")
    for name in ("recurrent_reg_fwd.cuh", "recurrent_wide_fwd.cuh"):
        text = (CSRC / name).read_text()
        call = re.search(r"reg_load_rows<[^;]*smem_u32\(wxs\)", text)
        assert call and "cluster_sync_all();" in text[call.end():text.index("auto run = ", call.end())], name
