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
