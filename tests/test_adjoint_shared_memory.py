"""The adjoint's solve adds in two ways through shared memory: block_sum (over a CTA, in a scratch array whose
first entries every warp writes on entry) and grid_total (over the CTAs, whose result all threads read after its
last barrier).  A block_sum may follow a grid_total with no barrier between, so their memory must not be the
same; the order is read from the source, since a race of this kind shows next to never."""

import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parents[1] / "cugal_b200" / "csrc" / "adjoint.cu"


def test_grid_total_does_not_return_block_sums_scratch():
    text = re.sub(r"//[^\n]*", "", SOURCE.read_text())
    body = text[text.index("double grid_total("):]
    body = body[:body.index("\n}\n")]
    returned = re.findall(r"return (\w+)", body)
    assert len(returned) == 1
    scratch = {a.strip() for a in re.findall(r"block_sum\([^,()]*,\s*(\w+)\)", text)}
    assert scratch and returned[0] not in scratch
    # its own variable, which a barrier at its start keeps until the total before has been read
    assert re.search(r"__shared__ double " + returned[0] + r";\s*__syncthreads\(\);", body)
