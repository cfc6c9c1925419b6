"""The backward pass of ragged_dot: both products in one native call, or one by one for everything else."""

import pytest
import torch

import gpu_ragged_dot_b200 as rd
from gpu_ragged_dot_b200 import ops

pytestmark = pytest.mark.gpu


def _inputs(m, k, n, dtype, trans, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    gs = torch.tensor([m // 3, 0, m - m // 3 - 2], dtype=torch.int32, device="cuda")
    x = torch.randn((m, k), device="cuda", generator=gen).to(dtype)
    A = torch.randn((3, n, k) if trans else (3, k, n), device="cuda", generator=gen).to(dtype)
    return x, A, gs, torch.randn((m, n), device="cuda", generator=gen).to(dtype)


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("m,k,n,dtype", [
    (200, 64, 136, torch.bfloat16),
    (171, 58, 77, torch.float16),   # rows that are not multiples of 16 bytes
    (150, 96, 132, torch.float32),
])
def test_backward_in_one_call(m, k, n, dtype, trans):
    x, A, gs, do = _inputs(m, k, n, dtype, trans)
    both = ops._native_backward(do, x, A, gs, trans)
    assert both is not None
    dx = ops.gmm_forward(do, A, gs, trans_rhs=not trans)
    dA = ops.tgmm_forward(do, x, gs) if trans else ops.tgmm_forward(x, do, gs)
    assert torch.equal(both[0], dx) and torch.equal(both[1], dA)
    xr, Ar = x.clone().requires_grad_(), A.clone().requires_grad_()
    # a cotangent with strides of its own, and either gradient alone
    wide = torch.cat([do, do], dim=1)[:, :n]
    for grads in (torch.autograd.grad(rd.ragged_dot(xr, Ar, gs, trans_rhs=trans), (xr, Ar), wide),
                  (torch.autograd.grad(rd.ragged_dot(xr, A, gs, trans_rhs=trans), xr, do)[0],
                   torch.autograd.grad(rd.ragged_dot(x, Ar, gs, trans_rhs=trans), Ar, do)[0])):
        assert torch.equal(grads[0], dx) and torch.equal(grads[1], dA)


def test_backward_of_other_forms(monkeypatch):
    x, A, gs, do = _inputs(200, 64, 136, torch.bfloat16, False)
    assert ops._native_backward(do, x, A.transpose(1, 2).contiguous().transpose(1, 2), gs, False) is None  # strided weights
    assert ops._native_backward(do, x, A, gs.long(), False) is None
    assert ops._native_backward(do, x[:, 1:].clone(), A[:, 1:].contiguous(), gs.cpu(), False) is None
    assert ops._native_backward(do.float(), x, A, gs, False) is None  # types that differ
    assert ops._native_backward(do[:-1], x, A, gs, False) is None     # rows that differ
    monkeypatch.setenv("RD_CHECK_STATUS", "1")
    assert ops._native_backward(do, x, A, gs, False) is None
    monkeypatch.delenv("RD_CHECK_STATUS")
    entry = dict(op="tgmm", k=64, n=136, g=3, tile_n=128)  # a tile table entry for one of the products
    monkeypatch.setattr(ops.tile_table, "_entries", [entry])
    assert ops._native_backward(do, x, A, gs, False) is None
    xr, Ar = x.clone().requires_grad_(), A.clone().requires_grad_()
    got = torch.autograd.grad(rd.ragged_dot(xr, Ar, gs), (xr, Ar), do)
    assert torch.equal(got[0], ops.gmm_forward(do, A, gs, trans_rhs=True)) and torch.equal(got[1], ops.tgmm_forward(x, do, gs))
