"""Kernels whose launch or tile depends on the size, at the edges of their tiles: against scipy, the
oracle, or FP64 torch."""

import numpy as np
import pytest
import torch
from scipy.optimize import linear_sum_assignment

from oracle import fugal_fp64 as O

pytestmark = pytest.mark.gpu


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _csr_graph(lengths, n, seed):
    """A symmetric graph whose first vertices have the given numbers of neighbours at least."""
    rng = np.random.default_rng(seed)
    e = rng.integers(0, n, size=(4 * n, 2))
    for v, d in enumerate(lengths):
        e = np.concatenate([e, np.stack([np.full(d, v), rng.permutation(n)[:d]], 1)])
    e = np.unique(np.sort(e[e[:, 0] != e[:, 1]], axis=1), axis=0)
    e = np.concatenate([e, e[:, ::-1]]).astype(np.int32)
    return torch.from_numpy(rng.permutation(e)).cuda()


@pytest.mark.parametrize("n", [1, 5, 149, 1000, 1001, 2049, 4100])
def test_adjoint_solve_matches_fp64(n):
    """The one-launch conjugate gradients (whole quads and odd rows) against a dense FP64 solve: the
    residual is below 1e-9 of the right side, so the gradient is exact to FP32 (2^-24, a few times)."""
    from cugal_b200.autograd import sinkhorn_adjoint
    P = torch.rand((n, n), generator=_gen(n), device="cuda") + 0.1
    for _ in range(30):
        P = P / P.sum(1, keepdim=True)
        P = P / P.sum(0, keepdim=True)
    G = torch.randn((n, n), generator=_gen(n + 1), device="cuda")
    dC, it, rel = sinkhorn_adjoint(P, G, 0.5, tol=1e-9)
    assert rel < 1e-9 and it >= 1
    Pd, Gd = P.double(), G.double()
    M = torch.zeros((2 * n, 2 * n), dtype=torch.float64, device="cuda")
    M[:n, :n] = M[n:, n:] = torch.eye(n, dtype=torch.float64, device="cuda")
    M[:n, n:], M[n:, :n] = Pd, Pd.T
    z = torch.cat([torch.ones(n, dtype=torch.float64), -torch.ones(n, dtype=torch.float64)]).cuda()[:, None] / (2 * n) ** 0.5
    a = torch.cat([(Gd * Pd).sum(1), (Gd * Pd).sum(0)])
    x = torch.linalg.solve(M + z @ z.T, a - z[:, 0] * (z[:, 0] @ a))
    ref = -2.0 * Pd * (Gd - x[:n, None] - x[None, n:])
    assert (dC.double() - ref).abs().max() < 1e-6 * max(float(ref.abs().max()), float(Pd.abs().max() * Gd.abs().max()))
