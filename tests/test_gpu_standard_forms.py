"""Which form of the scaling-form solve a call takes: the persistent one streams 16-byte pieces of K and of its
workspace, and whatever does not lie on such boundaries takes the form with launches, which reads single
numbers."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 300, 5000])
@pytest.mark.parametrize("offset", [8, 16, 24])
def test_workspace_off_a_16_byte_boundary(n, offset):
    """The same u and v to the FP32 sums' sqrt(n) 2^-24 of 30 updates (2e-5, as between the two forms)."""
    from cugal_b200 import _native as N
    K = torch.zeros((n, (n + 7) // 8 * 8), device="cuda")
    K[:, :n] = torch.exp(torch.rand((n, n), generator=torch.Generator(device="cuda").manual_seed(n), device="cuda") * -6)
    size = N.workspace_size("fugal_sinkhorn_standard_workspace_size", n)
    ws = torch.empty(size + 32, dtype=torch.uint8, device="cuda")
    got = []
    for base in (0, offset):
        u, v = (torch.full((n,), 1.0 / n, device="cuda") for _ in range(2))
        N.call("fugal_sinkhorn_standard_solve", K.data_ptr(), K.stride(0), n, u.data_ptr(), v.data_ptr(), 15, -1.0, 5,
               -1, None, ws.data_ptr() + base, size, N.stream_handle())
        got.append((u, v))
    for a, b in zip(*got):
        assert torch.allclose(a, b, rtol=2e-5, atol=0)


@pytest.mark.parametrize("n", [4, 7, 300, 2001, 16385])
def test_solve_holds_k_once_where_its_rows_need_no_padding(n):
    """Beside the cost a solve allocates K and, only where the persistent form needs 16-byte rows that K does not
    have, one padded copy; K comes back contiguous."""
    from cugal_b200.config import Config, SinkhornMethod
    from cugal_b200.sinkhorn import SinkhornState
    C = torch.rand((n, n), generator=torch.Generator(device="cuda").manual_seed(n), device="cuda")
    state = SinkhornState(n, Config(device="cuda", dtype=torch.float32, sinkhorn_method=SinkhornMethod.STANDARD,
                                    sinkhorn_regularization=0.5, sinkhorn_iterations=2))
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    K, _, _ = state.solve(C)
    torch.cuda.synchronize()
    peak = torch.cuda.max_memory_allocated() - before
    copies = 2 if n % 4 and n <= 16384 else 1
    assert peak <= copies * (n * (n + 7) * 4 + (1 << 21))  # torch rounds an allocation up by 2 MB at most
    assert K.is_contiguous() and K.shape == (n, n)
    assert torch.allclose(K, torch.exp(C * -2.0), rtol=1e-6, atol=0)
