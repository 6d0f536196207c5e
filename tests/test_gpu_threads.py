"""Two host threads, each on its own stream, on sizes that share a kernel but not its shared memory: the
launch of one never takes away the shared-memory limit that the other's larger launch needs, and every
result is the one of a call alone, bit for bit."""

import sys
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

CALLS = 150


def _config(**kw):
    from cugal_b200.config import Config, SinkhornMethod
    kw.setdefault("sinkhorn_method", SinkhornMethod.LOG)
    return Config(device="cuda", dtype=torch.float32, sinkhorn_threshold=0.0, sinkhorn_eval_freq=5, reabsorb_every=10,
                  **kw)


def _matrix(n):
    return torch.rand((n, n), generator=torch.Generator(device="cuda").manual_seed(n), device="cuda")


def _log(n, dtype=None, fixed=False):
    from cugal_b200.sinkhorn import SinkhornSolver, padded_ld
    cost = torch.zeros((n, padded_ld(n)), device="cuda")
    cost[:, :n] = _matrix(n) * -20
    s = SinkhornSolver(n, _config(sinkhorn_iterations=12, stream_dtype=dtype, polish_sweeps=1), "cuda")
    s.fixed_order = fixed
    u, v = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")

    def call():
        s.solve(cost, u, v)
        return u, v
    return call


def _standard(n):
    from cugal_b200.config import SinkhornMethod
    from cugal_b200.sinkhorn import StandardSolver, padded_ld
    K = torch.zeros((n, padded_ld(n)), device="cuda")
    K[:, :n] = torch.exp(_matrix(n) * -5)
    s = StandardSolver(n, _config(sinkhorn_iterations=12, sinkhorn_method=SinkhornMethod.STANDARD), "cuda")

    def call():
        u, v = torch.full((n,), 1.0 / n, device="cuda"), torch.full((n,), 1.0 / n, device="cuda")
        s.solve(K, u, v)
        return u, v
    return call


def _exact(n):
    from cugal_b200.exact_lap import exact_assign
    P = _matrix(n)
    P[torch.arange(n), torch.arange(n)] += 1.0  # one search step a row
    return lambda: exact_assign(P)


def _greedy(n):
    from cugal_b200.config import HungarianMethod
    from cugal_b200.greedy_lap import greedy_assign
    P = _matrix(n)
    return lambda: (greedy_assign(P.clone(), HungarianMethod.DOUBLE_GREEDY),)


def _matmul(n):
    from cugal_b200 import cuda_kernels
    M = _matrix(n).t()
    columns = torch.arange(n, dtype=torch.int32, device="cuda").roll(1)
    rows = torch.arange(n + 1, dtype=torch.int32, device="cuda")

    def call():
        out = torch.empty_like(M)
        cuda_kernels.adjacency_matmul(columns, rows, M, out, False)
        return (out,)
    return call


def _adjoint(n):
    from cugal_b200.autograd import sinkhorn_adjoint
    P = _matrix(n) / n
    P += torch.eye(n, device="cuda") * 0.5
    G = _matrix(n)
    return lambda: sinkhorn_adjoint(P, G, 0.3, max_iter=2)[:1]


@pytest.mark.parametrize("make,sizes", [
    (_log, (600, 1000)),
    (lambda n: _log(n, torch.bfloat16), (600, 1000)),
    (lambda n: _log(n, fixed=True), (600, 1000)),
    (_standard, (600, 1000)),
    (_exact, (600, 1000)),
    (_greedy, (600, 1000)),
    (_matmul, (600, 1000)),
    (_adjoint, (1000, 3000)),
], ids=["log", "log16", "log_cluster", "standard", "exact", "greedy", "matmul", "adjoint"])
def test_two_sizes_of_one_kernel_from_two_threads(make, sizes):
    alone = [tuple(t.clone() for t in make(n)()) for n in sizes]
    torch.cuda.synchronize()
    start = threading.Barrier(2)
    failed = [None, None]

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                call = make(sizes[k])
                torch.cuda.current_stream().synchronize()
                start.wait()
                for _ in range(CALLS):
                    got = call()
                for a, b in zip(alone[k], got):
                    assert torch.equal(a, b)
        except BaseException as exc:
            failed[k] = exc
            start.abort()

    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    torch.cuda.synchronize()
    for exc in failed:
        if exc is not None:
            raise exc
