"""Bounded waits of the persistent kernels over FP32 rows that run out: one copy of CTA 0 is armed for 16 bytes
more than it delivers (``FUGAL_TEST_FAULT_ROW_FP32``), every wait gives up after 1 ms
(``FUGAL_TEST_WAIT_LIMIT_NS``), all CTAs end, the status says so, and the same solve runs again afterwards.
n = 300: every row of a CTA stays in shared memory; 3000 and 5000: rows stream through it (column sums in
registers and in tensor memory)."""

import dataclasses

import pytest
import torch

pytestmark = pytest.mark.gpu


def _config(method):
    from cugal_b200.config import Config, SinkhornMethod
    return Config(device="cuda", dtype=torch.float32, sinkhorn_method=SinkhornMethod[method],
                  sinkhorn_regularization=0.5, sinkhorn_iterations=30, sinkhorn_threshold=0.0, sinkhorn_eval_freq=5)


def _cost(n):
    return torch.rand((n, n), generator=torch.Generator(device="cuda").manual_seed(n), device="cuda") * 5


@pytest.fixture
def unmet_copy(monkeypatch):
    def arm(row):
        monkeypatch.setenv("FUGAL_TEST_FAULT_ROW_FP32", str(row))
        monkeypatch.setenv("FUGAL_TEST_WAIT_LIMIT_NS", "1000000")

    def disarm():
        monkeypatch.delenv("FUGAL_TEST_FAULT_ROW_FP32")
        monkeypatch.delenv("FUGAL_TEST_WAIT_LIMIT_NS")
    return arm, disarm


@pytest.mark.parametrize("n,row", [(300, 0), (300, 2), (3000, 5), (5000, 1)])
def test_scaling_form(n, row, unmet_copy):
    from cugal_b200 import _native as N
    from cugal_b200.profile import SinkhornProfile
    from cugal_b200.sinkhorn import SinkhornState
    arm, disarm = unmet_copy
    cfg, C = _config("STANDARD"), _cost(n)
    _, u0, v0 = SinkhornState(n, cfg).solve(C)
    assert u0.isfinite().all() and v0.isfinite().all()
    arm(row)
    K, u, v = SinkhornState(n, cfg).solve(C)  # nobody reads the record: no half-iterated result
    assert u.isnan().all() and v.isnan().all() and K.isfinite().all()
    with pytest.raises(N.NativeError, match="device status 6"):
        SinkhornState(n, cfg).solve(C, profile=SinkhornProfile())
    disarm()
    _, u1, v1 = SinkhornState(n, cfg).solve(C)
    assert torch.equal(u0, u1) and torch.equal(v0, v1)


@pytest.mark.parametrize("n,row", [(300, 0), (300, 2), (3000, 5), (5000, 1)])
def test_log_form(n, row, unmet_copy):
    from cugal_b200 import _native as N
    from cugal_b200.profile import SinkhornProfile
    from cugal_b200.sinkhorn import SinkhornState
    arm, disarm = unmet_copy
    cfg, C = _config("LOG"), _cost(n)
    _, u0, v0 = SinkhornState(n, cfg).solve(C)
    arm(row)
    with pytest.raises(N.NativeError, match="device status 6"):
        SinkhornState(n, cfg).solve(C, profile=SinkhornProfile())
    disarm()
    _, u1, v1 = SinkhornState(n, cfg).solve(C)
    assert torch.equal(u0, u1) and torch.equal(v0, v1)


def test_16_bit_solve_after_fp32_sweeps_that_gave_up(unmet_copy):
    """The FP32 sweeps before the 16-bit ones give up: the sweeps and the polish that follow end as well."""
    from cugal_b200 import _native as N
    from cugal_b200.profile import SinkhornProfile
    from cugal_b200.sinkhorn import SinkhornState
    arm, disarm = unmet_copy
    cfg, C = dataclasses.replace(_config("LOG"), stream_dtype=torch.bfloat16, fp32_warmup_sweeps=2), _cost(3000)
    _, u0, v0 = SinkhornState(3000, cfg).solve(C)
    arm(1)
    with pytest.raises(N.NativeError, match="device status 6"):
        SinkhornState(3000, cfg).solve(C, profile=SinkhornProfile())
    disarm()
    _, u1, v1 = SinkhornState(3000, cfg).solve(C)
    assert torch.equal(u0, u1) and torch.equal(v0, v1)


@pytest.mark.parametrize("n", [100, 1000])
@pytest.mark.parametrize("barrier", [1, 2, 3, 4, 7])
def test_adjoint_solve(n, barrier, monkeypatch):
    """The last CTA's wait on a barrier runs out (``FUGAL_TEST_FAULT_BARRIER``) after it has arrived.  An
    iteration has three barriers, one comes before the first: with one iteration the fourth is the last, which
    all other CTAs pass."""
    from cugal_b200 import _native as N
    from cugal_b200.autograd import sinkhorn_adjoint
    P = torch.rand((n, n), generator=torch.Generator(device="cuda").manual_seed(n), device="cuda") / n
    P += torch.eye(n, device="cuda") * 0.5
    G = torch.rand((n, n), generator=torch.Generator(device="cuda").manual_seed(n + 1), device="cuda")
    kw = dict(tol=0.0, max_iter=(barrier + 1) // 3)
    dC, it, rel = sinkhorn_adjoint(P, G, 0.3, **kw)
    assert it == kw["max_iter"] and dC.isfinite().all()
    monkeypatch.setenv("FUGAL_TEST_FAULT_BARRIER", str(barrier))
    monkeypatch.setenv("FUGAL_TEST_WAIT_LIMIT_NS", "1000000")
    with pytest.raises(N.NativeError, match="device status 6"):
        sinkhorn_adjoint(P, G, 0.3, **kw)
    monkeypatch.delenv("FUGAL_TEST_FAULT_BARRIER")
    monkeypatch.delenv("FUGAL_TEST_WAIT_LIMIT_NS")
    again, _, _ = sinkhorn_adjoint(P, G, 0.3, **kw)
    assert torch.equal(dC, again)
