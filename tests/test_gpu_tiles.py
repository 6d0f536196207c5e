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


@pytest.mark.parametrize("n,lengths", [(5, [1]), (33, [31, 32]), (100, [30, 31, 32, 33, 34, 63, 64, 65]),
                                       (3000, [24, 32, 33, 1500, 2999]), (16385, [40, 9000])])
def test_graph_rows_at_register_and_memory_lengths(n, lengths):
    """CSR order, triangle counts (rows of up to 32 entries in registers, longer ones in memory, edges of
    one row over several warps), with and without 64-bit counts, and neighbour averages: bit for bit."""
    from cugal_b200.adjacency import Adjacency
    from cugal_b200.feature_extraction import average_neighbor_features, graph_features
    lengths = [d for d in lengths if d <= 8000]  # the row sort's limit
    A = Adjacency.from_edges(_csr_graph(lengths, n, n), n)
    rp, col = A.row_pointers.cpu().numpy(), A.col_indices.cpu().numpy()
    for r in range(n):
        assert np.all(np.diff(col[rp[r]:rp[r + 1]]) > 0)
    odeg, otri = O.triangle_counts(rp, col)
    deg, clust, dc, tc = graph_features(A, with_counts=True)
    assert np.array_equal(dc.cpu().numpy(), odeg) and np.array_equal(tc.cpu().numpy(), otri)
    deg2, clust2 = graph_features(A)
    assert torch.equal(deg, deg2) and torch.equal(clust, clust2)
    assert np.array_equal(clust.cpu().numpy(), O.clustering_from_counts(odeg, otri))
    avg = average_neighbor_features(A, clust).cpu().numpy()
    assert np.array_equal(avg, O.average_neighbor(rp, col, clust.cpu().numpy()))


@pytest.mark.parametrize("maximize", [True, False])
@pytest.mark.parametrize("n", [1, 2, 31, 1023, 1024, 1025, 2049, 4097])
def test_exact_lap_owned_columns(n, maximize):
    """Every number of owned columns per thread, with many ties (integers 0 .. 3, zeros of both signs)."""
    from cugal_b200.exact_lap import exact_assign
    rng = np.random.default_rng(n)
    P = np.zeros((n, n), dtype=np.float32)
    P[rng.random((n, n)) < 0.5] = -0.0
    rows = np.arange(n)
    for k in range(3):
        P[rows, rng.permutation(n)] += rng.integers(0, 4, size=n).astype(np.float32)
    cols, _, status = exact_assign(torch.tensor(P, device="cuda"), maximize=maximize)
    assert int(status.item()) == 0
    np.testing.assert_array_equal(cols.cpu().numpy(), linear_sum_assignment(P, maximize=maximize)[1])


def test_exact_lap_above_owned_columns():
    """8192 is the widest owned matrix, 8193 takes the kernel with its arrays in global memory."""
    from cugal_b200.exact_lap import exact_assign
    for n in (8192, 8193):
        g = _gen(n)
        perm = torch.randperm(n, generator=g, device="cuda")
        P = torch.rand((n, n), generator=g, device="cuda") * 1e-4
        P[torch.arange(n, device="cuda"), perm] += 1.0
        cols, steps, status = exact_assign(P)
        assert int(status.item()) == 0 and int(steps.item()) == n and torch.equal(cols, perm)


@pytest.mark.parametrize("ld_pad,offset", [(0, 0), (3, 0), (0, 1)])
@pytest.mark.parametrize("cols", [1, 3, 1023, 1024, 1028, 2052, 4100, 8192, 8196, 20001])
def test_log_step_widths(cols, ld_pad, offset):
    """Rows in registers (up to 8192 columns) and in pieces, 16-byte and scalar access: relative error of
    the FP32 LSE, at most a few ulp of the largest term plus the summation's sqrt(cols) 2^-24."""
    from cugal_b200 import _native as N
    rows, g = 37, _gen(cols)
    buf = torch.randn(offset + rows * (cols + ld_pad), generator=g, device="cuda") * 5
    K = buf[offset:].view(rows, cols + ld_pad)[:, :cols]
    add, out = torch.randn(cols, generator=g, device="cuda"), torch.randn(rows, generator=g, device="cuda")
    add[cols // 2:cols // 2 + 1] = float("-inf") if cols > 1 else 0.0
    old = out.clone()
    for w in (1.0, 0.6):
        out.copy_(old)
        N.call("fugal_sinkhorn_log_step", K.data_ptr(), rows, cols, K.stride(0), add.data_ptr(), out.data_ptr(), w,
               N.stream_handle())
        lse = torch.logsumexp(K.double() + add.double(), 1)
        ref = -lse if w == 1.0 else (1 - w) * old.double() - w * lse
        assert (out.double() - ref).abs().max() < 4e-6 * max(1.0, float(lse.abs().max()))


@pytest.mark.parametrize("n,ld_pad", [(1, 0), (3, 1), (1000, 0), (1000, 3), (1025, 0), (2052, 4)])
def test_elementwise_access(n, ld_pad):
    """regularize, add_distance, the log update, count_le and the marginals with whole 16-byte rows and
    without: the FP32 operations of the reference, bit for bit where it fixes them."""
    from cugal_b200 import _native as N
    from cugal_b200 import cuda_kernels as ck
    g = _gen(n + ld_pad)
    new = lambda s: (torch.randn((n, n + ld_pad), generator=g, device="cuda") * s)[:, :n]
    G, P, K = new(1.0), new(0.1).abs(), new(2.0) - 6
    fs, ft = (torch.rand((n, 4), generator=g, device="cuda") * 9 for _ in range(2))
    u, v = (torch.randn(n, generator=g, device="cuda") for _ in range(2))
    ref = G + (3.0 - 6.0 * P)
    ck.regularize(G, P, 3)
    assert torch.equal(G, ref)
    d = (fs[:, None, :] - ft[None, :, :]).square().double().sum(2).float().sqrt()
    out = G.clone()
    ck.add_distance(fs, ft, out)
    assert torch.equal(out, G + d)
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    N.call("fugal_count_le", P.data_ptr(), P.stride(0), n, 0.05, count.data_ptr(), N.stream_handle())
    assert int(count.item()) == int((P <= 0.05).sum())
    q = torch.exp(K.double() + v.double() + u.double()[:, None])
    assert abs(ck.sinkhorn_log_marginal(K, u, v) - float((q.sum(1) - 1).abs().sum())) < 1e-5 * float(q.sum() + n)
    err = torch.zeros(1, dtype=torch.float64, device="cuda")
    N.call("fugal_sinkhorn_log_marginal", K.data_ptr(), n, K.stride(0), u.data_ptr(), v.data_ptr(), 0, err.data_ptr(),
           N.stream_handle())
    assert abs(float(err.item()) - float((q.sum(0) - 1).abs().sum())) < 1e-5 * float(q.sum() + n)
    P2 = P.clone()
    gap = ck.update_quasi_permutation_log(P2, K, u, v, 0.3, 0.5)
    assert torch.allclose(P2.double(), P.double() + 0.3 * (q - P.double()), rtol=2e-6, atol=1e-7)
    terms = (q - P.double()) * K.double() * -0.5
    assert abs(gap - abs(float(terms.sum()))) < 1e-5 * float(terms.abs().sum())


@pytest.mark.parametrize("n", [1, 7, 1000, 14336, 14337, 28673])
def test_transposed_operand_rows(n):
    """4, 2 and 1 rows of the operand per CTA: the sums of the plain operand's kernel, in the same order."""
    from cugal_b200.adjacency import Adjacency
    A = Adjacency.from_edges(_csr_graph([], n, n), n)
    M = torch.rand((n, n), generator=_gen(n), device="cuda")
    expect = A.mul(M, negate_lhs=True)
    rows = torch.randint(0, n, (50,), device="cuda")
    got = A.mul(M.T.contiguous().T, negate_lhs=True)
    assert torch.equal(got[rows], expect[rows]) and torch.equal(got[:, rows], expect[:, rows])


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


@pytest.mark.parametrize("n", [1, 6, 150, 1025, 2050, 4097, 6143, 8190, 8193, 12289, 16387])
def test_standard_solve_widths(n):
    """The persistent scaling-form solve at the edges of its shapes (rows of odd widths included) and the
    launches above it, against FP64: u and v after 15 iterations to 2e-5, the FP32 sums' sqrt(n) 2^-24 of
    30 updates that do not amplify them."""
    from cugal_b200.config import Config, SinkhornMethod
    from cugal_b200.profile import SinkhornProfile
    from cugal_b200.sinkhorn import SinkhornState
    C = torch.rand((n, n), generator=_gen(n), device="cuda") * 3
    cfg = Config(device="cuda", dtype=torch.float32, sinkhorn_method=SinkhornMethod.STANDARD,
                 sinkhorn_regularization=0.5, sinkhorn_iterations=15, sinkhorn_threshold=-1.0, sinkhorn_eval_freq=5)
    prof = SinkhornProfile()
    K, u, v = SinkhornState(n, cfg).solve(C, cfg, prof)
    assert prof.iteration_count == 15 and K.is_contiguous()
    Kd = K.double()
    errors = []
    ue = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    for t in range(15):
        ve = 1 / (ue @ Kd + 1e-16)
        ue = 1 / (Kd @ ve + 1e-16)
        if t % 5 == 0:
            errors.append(float(((ue @ Kd) * ve - 1).abs().sum()))
    assert torch.allclose(u.double(), ue, rtol=2e-5, atol=0) and torch.allclose(v.double(), ve, rtol=2e-5, atol=0)
    np.testing.assert_allclose(prof.errors, errors, rtol=1e-2, atol=1e-6 * n)


@pytest.mark.parametrize("n", [150, 2050, 6143, 12289])
def test_standard_momentum_matches_the_launches(n):
    """Momentum (and rows whose last quad holds NaN past n) in the persistent form against the form with
    launches, which unaligned rows take: the same FP32 updates, to 2e-5."""
    from cugal_b200 import _native as N
    from cugal_b200.sinkhorn import exp_scale, read_record
    C = torch.rand((n, n), generator=_gen(n), device="cuda") * 3
    ws = torch.empty(N.workspace_size("fugal_sinkhorn_standard_workspace_size", n), dtype=torch.uint8, device="cuda")
    got = []
    for ld in ((n + 7) // 8 * 8, n + 1 if (n + 1) % 4 else n + 2):
        K = torch.full((n, ld), float("nan"), device="cuda")
        exp_scale(C, -2.0, K)
        u = torch.full((n,), 1.0 / n, device="cuda")
        v = u.clone()
        rec = torch.empty(N.RECORD_BYTES, dtype=torch.uint8, device="cuda")
        N.call("fugal_sinkhorn_standard_solve", K.data_ptr(), ld, n, u.data_ptr(), v.data_ptr(), 15, -1.0, 5, 5,
               rec.data_ptr(), ws.data_ptr(), ws.numel(), N.stream_handle())
        got.append((u, v, read_record(rec.cpu())))
    (u1, v1, r1), (u2, v2, r2) = got
    assert r1.iteration_count == r2.iteration_count == 15
    assert torch.allclose(u1, u2, rtol=2e-5, atol=0) and torch.allclose(v1, v2, rtol=2e-5, atol=0)
