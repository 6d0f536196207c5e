"""Tensor memory orders a load after a store of the same thread only through a wait on the stores
(tcgen05.wait::st).  The sweep kernels keep running column sums there: every row loads, adds and stores
them, so a wait has to lie between the stores of one row and the loads of the next, and between the last
row and the read-out.  The order is read from the source: a missing wait gives wrong sums only now and then."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cugal_b200" / "csrc"


def _code(name):
    text = (CSRC / name).read_text()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def _block(text, start):
    """(body, end) of the braces that open at or after ``start``."""
    begin = text.index("{", start)
    depth = 0
    for k in range(begin, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[begin + 1:k], k
    raise AssertionError("unbalanced braces")


def _kernel(name, kernel):
    """(body of the row loop, what follows it) of a sweep kernel."""
    text = _code(name)
    body, _ = _block(text, re.search(r"\b" + kernel + r"\(", text).end())
    loop = re.search(r"for \([^)]*;\s*r < nrows;", body)
    rows, end = _block(body, loop.end())
    return rows, body[end:]


def _first(text, pattern):
    m = re.search(pattern, text)
    assert m is not None, pattern
    return m.start()


@pytest.mark.parametrize("name,kernel", [("sinkhorn_rows.cu", "rows_kernel"),
                                         ("sinkhorn_standard.cu", "std_rows_kernel")])
def test_persistent_kernels_wait_for_the_stores_of_the_row_before(name, kernel):
    rows, after = _kernel(name, kernel)
    wait, access = r"cols\.settle\(\)", r"cols\.(add|total)\("
    assert wait.replace("\\", "") in rows and _first(rows, wait) < _first(rows, access)
    assert wait.replace("\\", "") in after and _first(after, wait) < _first(after, access)


def test_settle_waits_where_the_sums_are_in_tensor_memory():
    state = _code("sinkhorn_rows.cuh")
    body, _ = _block(state, state.index("struct ColumnState<EPT, false>"))
    settle, _ = _block(body, _first(body, r"void settle\(\)"))
    assert "tmem_wait_st()" in settle
    assert "tmem_st16(tsum" in body and "tmem_ld16(tsum" in body


def test_row_sweep_waits_for_the_stores_of_the_row_before():
    rows, after = _kernel("sinkhorn.cu", "row_sweep_kernel")
    for part in (rows, after):
        assert "tmem_wait_st()" in part and _first(part, r"tmem_wait_st\(\)") < _first(part, r"tmem_ld16\(tcol")
