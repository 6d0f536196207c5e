"""A stage of the sweep kernels' rings is read by the threads of a row (generic proxy) and then refilled by a bulk
copy (async proxy).  The barrier between orders the threads; accesses of two proxies to the same shared memory are
ordered by a proxy fence of the thread that issues the copy.  Read from the source, as the copy takes far longer
to arrive than the reads that it must not overtake."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cugal_b200" / "csrc"


@pytest.mark.parametrize("name,refill", [
    ("sinkhorn.cu", "issue(bt + p.stages, s);"), ("sinkhorn.cu", "issue(u, si);"),
    ("sinkhorn_rows.cu", "issue(row, s, ph ^ 1u, false);"), ("sinkhorn_standard.cu", "issue(row, s, ph ^ 1u, false);")])
def test_refill_follows_a_proxy_fence(name, refill):
    """The fence stands in the same branch as the refill, which is taken by one thread after a barrier."""
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    assert text.count(refill) == 1
    before = text[:text.index(refill)]
    branch = before[before.rindex("if (tid == 0" if "tid == 0" in before[-700:] else "if (gt == 0"):]
    assert "fence_proxy_async_smem();" in branch
