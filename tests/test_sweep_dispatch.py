"""Which kernel runs the sweeps of a size and stream type, at both sides of every limit (no GPU needed)."""

import pytest

from cugal_b200 import _native as N


@pytest.mark.parametrize("n,dtype,kernel", [
    (1, N.FUGAL_F32, "rows_kernel"), (8192, N.FUGAL_F32, "rows_kernel"), (8193, N.FUGAL_F32, "sweep_kernel"),
    (32768, N.FUGAL_F32, "sweep_kernel"),
    (1, N.FUGAL_BF16, "rows_kernel"), (24576, N.FUGAL_BF16, "rows_kernel"), (24577, N.FUGAL_BF16, "row_sweep_kernel"),
    (65536, N.FUGAL_BF16, "row_sweep_kernel"), (65537, N.FUGAL_BF16, "sweep_kernel"),
    (24576, N.FUGAL_F16, "rows_kernel"), (24577, N.FUGAL_F16, "row_sweep_kernel"),
])
def test_kernel_of_the_sweeps(n, dtype, kernel):
    assert N.sweep_kernel(n, dtype) == kernel


def test_environment_and_bad_arguments(monkeypatch):
    for n, dtype in ((0, N.FUGAL_F32), (-5, N.FUGAL_BF16), (100, 7)):
        assert N.sweep_kernel(n, dtype) is None
    monkeypatch.setenv("FUGAL_ROW_SWEEP", "0")  # 16-bit sweeps by the cluster kernel
    assert N.sweep_kernel(300, N.FUGAL_BF16) == N.sweep_kernel(32768, N.FUGAL_BF16) == "sweep_kernel"
    assert N.sweep_kernel(300, N.FUGAL_F32) == "rows_kernel"
    monkeypatch.setenv("FUGAL_SWEEP_SHAPE", "256x16")  # a shape of the cluster kernel asked for by name
    assert N.sweep_kernel(300, N.FUGAL_F32) == "sweep_kernel"


@pytest.mark.parametrize("dtype", [N.FUGAL_F32, N.FUGAL_BF16, N.FUGAL_F16])
@pytest.mark.parametrize("n", [0, -1])
def test_plan_info_refuses_sizes_below_one(n, dtype):
    with pytest.raises(N.NativeError, match="bad shape"):
        N.sinkhorn_plan(n, dtype)
