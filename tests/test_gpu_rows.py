"""The row-owned persistent Sinkhorn sweeps (csrc/sinkhorn_rows.cu) against FP64, at the edges of
their launch shapes: the largest size of each (streams, columns per thread) pair and one more,
sizes below one row per CTA, rows that stay in shared memory and rows that stream through it,
and two solves in flight on two streams.

Tolerance of the FP32 solves: the exponents are up to about 115 in base 2 (costs of 80 nats),
rounded to 2^-18 (3.8e-6); a row or column update averages such errors, and T = 24 updates of
either kind add at most 2 T 3.8e-6 = 1.8e-4 to a dual.  BF16 and FP16 streams: the plans are
within 1e-2 and 2e-3 after the FP32 polish sweep, as in the other reduced-precision tests."""

import threading

import pytest
import torch

from oracle import fugal_torch64 as T

pytestmark = pytest.mark.gpu

ITERATIONS = 24


def _cost(n, seed):
    from cugal_b200.sinkhorn import padded_ld
    g = torch.Generator(device="cuda").manual_seed(seed)
    cost = torch.zeros((n, padded_ld(n)), device="cuda")
    cost[:, :n] = torch.rand((n, n), generator=g, device="cuda") * -80
    return cost


def _solver(n, dtype, iterations=ITERATIONS, momentum=None):
    from cugal_b200.config import Config, SinkhornMethod
    from cugal_b200.sinkhorn import SinkhornSolver
    return SinkhornSolver(n, Config(device="cuda", dtype=torch.float32, sinkhorn_method=SinkhornMethod.LOG,
                                    sinkhorn_iterations=iterations, sinkhorn_threshold=0.0, sinkhorn_eval_freq=5,
                                    stream_dtype=dtype, reabsorb_every=10, sinkhorn_momentum_start=momentum), "cuda")


def _solve(n, dtype, cost, fixed=False, **kw):
    s = _solver(n, dtype, **kw)
    s.fixed_order = fixed
    u, v = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
    s.solve(cost, u, v)
    torch.cuda.synchronize()
    return u.double(), v.double()


def _exact(n, cost, iterations=ITERATIONS):
    u = torch.zeros(n, dtype=torch.float64, device="cuda")
    v = torch.zeros_like(u)
    T.sinkhorn_log_solve_(cost[:, :n].double(), u, v, iterations, 0.0, 5, block=1024)
    return u, v


@pytest.mark.parametrize("n", [1, 2, 17, 147, 149, 1024, 1025, 2048, 2049, 4096, 4097, 6144, 6145, 8192])
def test_fp32_matches_fp64(n):
    cost = _cost(n, n)
    u, v = _solve(n, None, cost)
    ue, ve = _exact(n, cost)
    assert (u - ue).abs().max() < 1.8e-4 and (v - ve).abs().max() < 1.8e-4


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 1e-2), (torch.float16, 2e-3)])
@pytest.mark.parametrize("n", [3, 150, 1024, 2049, 4097, 6145, 8193, 12289, 16385, 24576])
def test_16_bit_stream_matches_fp64(n, dtype, tol):
    cost = _cost(n, n)
    u, v = _solve(n, dtype, cost)
    ue, ve = _exact(n, cost)
    for r0 in range(0, n, 4096):
        K = cost[r0:r0 + 4096, :n].double()
        d = torch.exp(K + u[r0:r0 + 4096, None] + v) - torch.exp(K + ue[r0:r0 + 4096, None] + ve)
        assert d.abs().max() < tol


@pytest.mark.parametrize("n", [300, 2500, 5000])
def test_momentum_and_fixed_order(n):
    """Momentum (the exact path) and the order of sums fixed by the caller: the same solve."""
    cost = _cost(n, n + 1)
    a, b = _solve(n, None, cost, momentum=5), _solve(n, None, cost, fixed=True, momentum=5)
    assert (a[0] - b[0]).abs().max() < 3.6e-4 and (a[1] - b[1]).abs().max() < 3.6e-4


def test_two_solves_in_flight():
    """Two host threads, each on its own stream: the grid barriers of one solve never wait for the other's."""
    sizes = (700, 3000)
    alone = [_solve(n, None, _cost(n, n), iterations=200) for n in sizes]
    got = [None, None]

    def work(k):
        n = sizes[k]
        with torch.cuda.stream(torch.cuda.Stream()):
            cost, s = _cost(n, n), _solver(n, None, iterations=200)
            u, v = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
            for _ in range(20):
                s.solve(cost, u, v)
            torch.cuda.current_stream().synchronize()
            got[k] = (u.double(), v.double())

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, got):
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
