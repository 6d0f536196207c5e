"""A 16-bit solve in which a wait ran out (``FUGAL_TEST_FAULT_ROW``: a copy that never completes) ends without
its FP32 polish sweeps: their grid barrier counts arrivals, and a CTA that gave up has not arrived."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [512, 3000])
def test_no_polish_after_a_wait_ran_out(n, monkeypatch):
    from cugal_b200 import _native as N
    from cugal_b200.config import Config, SinkhornMethod
    from cugal_b200.sinkhorn import SinkhornSolver, padded_ld
    cost = torch.zeros((n, padded_ld(n)), device="cuda")
    cost[:, :n] = torch.rand((n, n), generator=torch.Generator(device="cuda").manual_seed(n), device="cuda") * -20
    s = SinkhornSolver(n, Config(device="cuda", dtype=torch.float32, sinkhorn_method=SinkhornMethod.LOG,
                                 sinkhorn_iterations=20, sinkhorn_threshold=0.0, sinkhorn_eval_freq=5,
                                 stream_dtype=torch.bfloat16, polish_sweeps=2), "cuda")
    u, v = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
    rec = torch.empty(N.RECORD_BYTES, dtype=torch.uint8, device="cuda")

    def record():
        s.solve(cost, u, v, rec.data_ptr())
        return N.SolveRecord.from_buffer_copy(rec.cpu().numpy().tobytes())

    r = record()
    assert r.status == 0 and r.polish_count == 2
    good = u.clone(), v.clone()
    monkeypatch.setenv("FUGAL_TEST_FAULT_ROW", "1")
    monkeypatch.setenv("FUGAL_TEST_WAIT_LIMIT_NS", "1000000")
    r = record()
    assert r.status == 6 and r.polish_count == 0
    monkeypatch.delenv("FUGAL_TEST_FAULT_ROW")
    monkeypatch.delenv("FUGAL_TEST_WAIT_LIMIT_NS")
    r = record()
    assert r.status == 0 and r.polish_count == 2
    assert torch.equal(u, good[0]) and torch.equal(v, good[1])
