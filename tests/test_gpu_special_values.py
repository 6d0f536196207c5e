"""Infinities, NaN and the lowest FP32 value through the reference-compatible log-domain step, one row per case,
with the special entries in every 8192-column piece of a long row: as torch has it, whatever piece they are in."""

import pytest
import torch

pytestmark = pytest.mark.gpu

INF, NAN, LOW = float("inf"), float("nan"), torch.finfo(torch.float32).min


@pytest.mark.parametrize("cols", [5, 1024, 8192, 8200, 8201, 20000])
@pytest.mark.parametrize("piece", [0, 1, 2])
def test_log_step(cols, piece):
    from cugal_b200 import cuda_kernels
    first = piece * 8192
    if first >= cols:
        pytest.skip("no such piece")
    last = min(cols, first + 8192)
    K = torch.rand((9, cols), generator=torch.Generator(device="cuda").manual_seed(cols), device="cuda") * -5
    K[1, first:last] = -INF
    K[2, first:last] = LOW
    K[3, first] = NAN
    K[4, first:last] = -INF
    K[4, first] = NAN
    K[5] = -INF
    K[6] = -INF
    K[6, last - 1] = -2.0
    K[7] = LOW
    K[8, last - 1] = NAN
    add = torch.linspace(-1, 1, cols, device="cuda")
    out = torch.zeros(9, device="cuda")
    cuda_kernels.sinkhorn_log_step(K, add, out, 1.0)
    exact = -torch.logsumexp(K.double() + add.double(), 1)
    assert torch.equal(out.isnan(), exact.isnan()) and torch.equal(out.isinf(), exact.isinf())
    fine = exact.isfinite()
    # x + add rounds to 2^-24 of up to 6, the sums of up to 20000 FP32 exponentials to sqrt(n) 2^-24: 1e-5;
    # LOW + add keeps LOW, whose logarithm of a sum is LOW itself in FP32
    assert torch.allclose(out[fine].double(), exact[fine], rtol=1e-6, atol=1e-5)
