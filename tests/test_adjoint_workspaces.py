"""Workspaces of the two adjoints: each asks for the partial sums that its own kernels write, and the
unrolled step runs in any workspace from the matrix-vector product's size up."""

import pytest
import torch

from cugal_b200 import _native as N


def _partials(n, rows):
    return (-(-n // 1024) - (-n // rows)) * n * 8 + 256


@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000, 4096, 16384, 32768, 65536])
def test_matvec_asks_for_its_own_partials(n):
    """Blocks of 64 rows: 139 MB at n = 32768, not n^2 bytes."""
    assert N.workspace_size("fugal_plan_matvec_workspace_size", n) == _partials(n, 64)


@pytest.mark.parametrize("n,rows", [(1, 8), (1024, 8), (4096, 8), (4097, 16), (8192, 16), (8193, 32), (16384, 32),
                                    (16385, 64), (65536, 64)])
def test_unrolled_step_asks_for_at_most_512_partial_rows(n, rows):
    assert N.workspace_size("fugal_sinkhorn_unrolled_workspace_size", n) == _partials(n, rows)


def test_unrolled_workspace_rejects_bad_sizes():
    for n in (0, -1, 2**31):
        with pytest.raises(N.NativeError):
            N.workspace_size("fugal_sinkhorn_unrolled_workspace_size", n)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 70, 1025, 4097])
def test_unrolled_step_in_every_workspace(n):
    """The same gK, bit for bit, and the same reductions up to the order of at most n FP64 terms of one
    sign (relative error n 2^-53 each way) whatever the number of rows in a block."""
    g = torch.Generator(device="cuda").manual_seed(n)
    K = torch.rand((n, n), generator=g, device="cuda") * -5
    u, v = (torch.rand(n, generator=g, device="cuda") for _ in range(2))
    grad = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    for axis in (0, 1):
        results = []
        for rows in (8, 16, 32, 64):
            ws = torch.empty(_partials(n, rows), dtype=torch.uint8, device="cuda")
            gK, other = torch.ones_like(K), torch.zeros_like(grad)
            N.call("fugal_sinkhorn_unrolled_step_backward", K.data_ptr(), n, n, u.data_ptr(), v.data_ptr(),
                   grad.data_ptr(), axis, gK.data_ptr(), n, other.data_ptr(), ws.data_ptr(), ws.numel(),
                   N.stream_handle())
            results.append((gK, other))
        E = torch.exp(K.double() + (u[:, None] + v[None, :] if axis else v[:, None] + u[None, :]).double())
        exact = -(grad[:, None] * E).sum(0) if axis else -(E * grad[None, :]).sum(1)
        for gK, other in results:
            assert torch.equal(gK, results[0][0])
            assert torch.allclose(other, results[0][1], rtol=2 * n * 2.0**-53, atol=0)
            # the duals are added in FP32 or FP64: 2 roundings of values up to 2
            assert torch.allclose(other, exact, rtol=4 * 2.0**-23, atol=0)
        with pytest.raises(N.NativeError, match="too small"):
            N.call("fugal_sinkhorn_unrolled_step_backward", K.data_ptr(), n, n, u.data_ptr(), v.data_ptr(),
                   grad.data_ptr(), axis, gK.data_ptr(), n, other.data_ptr(), ws.data_ptr(),
                   _partials(n, 64) - 1, N.stream_handle())


def test_unrolled_gradient_vectors_come_in_blocks():
    """A long segment between checkpoints holds a few gradient vectors at a time, each zero, its own, and on
    a 256-byte boundary."""
    from cugal_b200.autograd import _zero_vectors
    k = -1
    for k, g in enumerate(_zero_vectors(1000, 5, 64, "cpu")):
        assert g.shape == (5,) and g.dtype == torch.float64 and not g.any() and g.storage_offset() * 8 % 256 == 0
        g += 1.0
        assert g.untyped_storage().nbytes() <= 32 * 64 * 8
    assert k == 999
