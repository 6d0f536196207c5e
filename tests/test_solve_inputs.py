"""What ``SinkhornState.solve`` takes as a cost, on the CPU: the kernel that forms the absorbed cost is
replaced by its arithmetic on the pointers that it is given, the solve itself by nothing."""

import ctypes
import dataclasses

import numpy as np
import pytest
import torch
from torch.autograd import forward_ad

from cugal_b200 import _native as N
from cugal_b200 import sinkhorn
from cugal_b200.config import Config, SinkhornMethod

REG = 0.25  # a power of two: a division and a product with its reciprocal round alike


def _array(pointer, ctype, shape):
    return np.ctypeslib.as_array(ctypes.cast(pointer, ctypes.POINTER(ctype)), shape=shape)


def _absorb(name, C, ldc, n, scale, U, V, K, ldk, cost, ld, stream):
    assert name == "fugal_absorb_cost"
    k = np.float32(scale) * _array(C, ctypes.c_float, (n, ldc))[:, :n]
    if K is not None:
        _array(K, ctypes.c_float, (n, ldk))[:, :n] = k
    out = _array(cost, ctypes.c_float, (n, ld))
    out[:, :n] = k.astype(np.float64) + _array(U, ctypes.c_double, (n, 1)) + _array(V, ctypes.c_double, (n,))
    out[:, n:] = 0.0


class _NoSolve:
    def solve(self, *args):
        pass


@pytest.fixture
def state(monkeypatch):
    """A state of 5 nodes with its duals on the CPU, zero increments, and no kernels."""
    n = 5
    s = object.__new__(sinkhorn.SinkhornState)
    s.n, s.method = n, SinkhornMethod.LOG
    s.config = Config(device="cpu", dtype=torch.float32, sinkhorn_method=SinkhornMethod.LOG,
                      sinkhorn_regularization=REG)
    s.U = torch.linspace(-1, 1, n, dtype=torch.float64)
    s.V = torch.linspace(3, -2, n, dtype=torch.float64)
    s._solver, s._rec = _NoSolve(), torch.empty(0)
    s._du, s._dv = torch.zeros(n), torch.zeros(n)
    monkeypatch.setattr(N, "require_cuda", lambda *args: None)
    monkeypatch.setattr(N, "stream_handle", lambda *args: 0)
    monkeypatch.setattr(N, "call", _absorb)
    return s


def _expected(C, s):
    K = -C / REG
    cost = torch.zeros(s.n, s.n)
    cost[:] = (K.double() + s.U[:, None] + s.V[None, :]).float().detach()
    return K, cost


def _check(s, C, K):
    expected, cost = _expected(C, s)
    assert K.dtype == torch.float32 and torch.equal(K.detach(), expected.detach().float())
    assert torch.equal(s._cost32[:, :s.n], cost)


def test_row_major_cost(state):
    C = torch.rand(5, 5)
    K, u, v = state.solve(C)
    _check(state, C, K)


def test_cost_on_another_device_is_refused(state, monkeypatch):
    state.U = state.U.to("meta")
    monkeypatch.setattr(N, "call", lambda *args: pytest.fail("a kernel was given another device's pointers"))
    with pytest.raises(RuntimeError):
        state.solve(torch.rand(5, 5))


def test_returned_kernel_keeps_the_tangent_of_the_cost(state):
    C, dC = torch.rand(5, 5), torch.rand(5, 5)
    with forward_ad.dual_level():
        K, _, _ = state.solve(forward_ad.make_dual(C, dC))
        tangent = forward_ad.unpack_dual(K).tangent
        assert tangent is not None and torch.equal(tangent, -dC / REG)
    _check(state, C, K)


def test_returned_kernel_keeps_the_graph_of_the_cost(state):
    C = torch.rand(5, 5, requires_grad=True)
    K, _, _ = state.solve(C)
    _check(state, C, K)
    (g,) = torch.autograd.grad(K.sum(), C)
    assert torch.equal(g, torch.full((5, 5), -1 / REG))
    with torch.no_grad():
        assert not state.solve(C)[0].requires_grad


@pytest.mark.parametrize("shape", [(5, 5), (1, 5), (5, 1), (5,), (1,), (), (1, 5, 5), (1, 1, 5, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_costs_that_broadcast(state, shape, dtype):
    """What K + u_i + v_j broadcasts to n x n is a cost, as in the reference's arithmetic; K keeps its shape."""
    C = torch.rand(shape).to(dtype)
    K, _, _ = state.solve(C)
    assert K.shape == torch.Size(shape)
    _check(state, C.float(), K)


@pytest.mark.parametrize("shape", [(4, 4), (5, 4), (2, 5, 5), (5, 5, 1), (6,)])
def test_other_shapes_are_refused(state, shape, monkeypatch):
    monkeypatch.setattr(N, "call", lambda *args: pytest.fail("a kernel was given a cost of another size"))
    with pytest.raises(RuntimeError):
        state.solve(torch.rand(shape))


@pytest.mark.parametrize("order", ["transposed", "columns", "steps", "repeated"])
def test_strides(state, order):
    base = torch.rand(10, 10)
    C = {"transposed": base[:5, :5].t(), "columns": base[:5, 2:7], "steps": base[::2, ::2],
         "repeated": base[0, :5].expand(5, 5)}[order]
    K, _, _ = state.solve(C)
    _check(state, C, K)


def test_negated_view(state):
    C = torch._neg_view(torch.rand(5, 5))
    K, _, _ = state.solve(C)
    _check(state, C.resolve_neg(), K)


def test_subclass_and_regularization_of_another_type(state):
    class Cost(torch.Tensor):
        pass
    C = torch.rand(5, 5).as_subclass(Cost)
    assert type(state.solve(C)[0]) is Cost
    C = torch.rand(5, 5)
    for reg in (torch.tensor(REG), np.float32(REG), torch.full((5, 1), REG)):
        K, _, _ = state.solve(C, dataclasses.replace(state.config, sinkhorn_regularization=reg))
        _check(state, C, K)
