"""The row-owned 16-bit sweep with a launch per sweep (rows of 24577 to 65536 columns): both stream types with
padded columns against FP64 at the smallest width, at an odd one and at one that takes two CTAs a row, and a wait
that runs out.

Tolerance: the plans of a BF16 and an FP16 stream are within 1e-2 and 2e-3 of FP64's after the FP32 polish
sweep, as in the other reduced-precision tests."""

import pytest
import torch

from oracle import fugal_torch64 as T

pytestmark = pytest.mark.gpu

ITERATIONS = 12


def _setup(n, dtype):
    from cugal_b200 import _native as N
    from cugal_b200.config import Config, SinkhornMethod
    from cugal_b200.sinkhorn import SinkhornSolver, padded_ld
    assert N.sweep_kernel(n, N.STREAM_DTYPES[dtype]) == "row_sweep_kernel"
    cost = torch.zeros((n, padded_ld(n)), device="cuda")
    cost[:, :n] = torch.rand((n, n), generator=torch.Generator(device="cuda").manual_seed(n), device="cuda") * -60
    s = SinkhornSolver(n, Config(device="cuda", dtype=torch.float32, sinkhorn_method=SinkhornMethod.LOG,
                                 sinkhorn_iterations=ITERATIONS, sinkhorn_threshold=0.0, sinkhorn_eval_freq=5,
                                 stream_dtype=dtype, reabsorb_every=10), "cuda")
    rec = torch.empty(N.RECORD_BYTES, dtype=torch.uint8, device="cuda")

    def solve():
        u, v = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
        s.solve(cost, u, v, rec.data_ptr())
        r = N.SolveRecord.from_buffer_copy(rec.cpu().numpy().tobytes())
        return u, v, r
    return cost, solve


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 1e-2), (torch.float16, 2e-3)])
@pytest.mark.parametrize("n", [24577, 30001, 33001])
def test_matches_fp64(n, dtype, tol):
    cost, solve = _setup(n, dtype)
    u, v, r = solve()
    assert r.status == 0 and r.iteration_count == ITERATIONS
    ue = torch.zeros(n, dtype=torch.float64, device="cuda")
    ve = torch.zeros_like(ue)
    T.sinkhorn_log_solve_(cost[:, :n].double(), ue, ve, ITERATIONS, 0.0, 5, block=1024)
    for r0 in range(0, n, 4096):
        K = cost[r0:r0 + 4096, :n].double()
        d = torch.exp(K + u[r0:r0 + 4096, None].double() + v.double())
        d -= torch.exp(K + ue[r0:r0 + 4096, None] + ve)
        assert d.abs().max() < tol


@pytest.mark.parametrize("n", [24577, 33001])
def test_wait_that_runs_out(n, monkeypatch):
    _, solve = _setup(n, torch.float16)
    u0, v0, r = solve()
    assert r.status == 0
    monkeypatch.setenv("FUGAL_TEST_FAULT_ROW", "1")
    monkeypatch.setenv("FUGAL_TEST_WAIT_LIMIT_NS", "1000000")
    assert solve()[2].status == 6
    monkeypatch.delenv("FUGAL_TEST_FAULT_ROW")
    monkeypatch.delenv("FUGAL_TEST_WAIT_LIMIT_NS")
    u1, v1, r = solve()
    assert r.status == 0 and torch.equal(u0, u1) and torch.equal(v0, v1)
