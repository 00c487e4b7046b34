"""Sharding by (batch, KV head): the pieces of a call give the bits of the whole call, also where the whole fills the GPU and
a piece does not. (Enough query rows in every piece that its forward does not take the split-key branch, whose split
count depends on batch and heads.)"""
import pytest
import torch

from flagattention_b200 import flash_attention, piecewise_attention
from flagattention_b200.sharding import shard
from gpu_util import make_qkv

pytestmark = pytest.mark.gpu


def _grads(q, k, v, do, causal):
    leaves = [t.detach().requires_grad_() for t in (q, k, v)]
    o = flash_attention(*leaves, causal)
    return (o.detach(),) + torch.autograd.grad(o, leaves, do)


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("B,Hq,Hkv,M,N,D,causal,dtype", [
    (16, 8, 2, 512, 512, 128, True, torch.bfloat16), (8, 32, 8, 1024, 1024, 128, True, torch.bfloat16),
    (4, 8, 1, 2048, 2048, 128, True, torch.bfloat16), (40, 8, 2, 512, 512, 64, True, torch.float16),
    (16, 16, 4, 1024, 1024, 64, False, torch.bfloat16), (6, 16, 2, 700, 1300, 32, True, torch.float16),
    (12, 4, 1, 600, 600, 16, False, torch.float16), (80, 24, 1, 65, 129, 128, True, torch.float16),
])
def test_pieces_give_the_bits_of_the_whole(B, Hq, Hkv, M, N, D, causal, dtype, deterministic):
    q, k, v, do = make_qkv(B, Hq, Hkv, M, N, D, dtype, seed=5)
    torch.use_deterministic_algorithms(deterministic)
    try:
        whole = _grads(q, k, v, do, causal)
        for rank in (0, 3):
            # pieces of the inputs beside the pieces of the whole call's results
            inputs = shard(q, k, v, rank, 4, do)
            results = shard(whole[0], whole[2], whole[3], rank, 4, whole[1])
            for (qp, kp, vp, dop), (o, dk, dv, dq) in list(zip(inputs, results))[:2]:
                got = _grads(qp, kp, vp, dop, causal)
                assert torch.equal(got[0], o) and torch.equal(got[2], dk) and torch.equal(got[3], dv)
                if deterministic:  # (dQ is otherwise summed in no fixed order)
                    assert torch.equal(got[1], dq)
    finally:
        torch.use_deterministic_algorithms(False)


def test_piecewise_pieces():
    inputs = [torch.randn(64, 2, 700, 64, device="cuda", dtype=torch.bfloat16) for _ in range(5)]
    do = torch.randn_like(inputs[0])

    def grads(rows):
        leaves = [t[rows].clone().requires_grad_() for t in inputs]
        return torch.autograd.grad(piecewise_attention(*leaves, 256, causal=True), leaves, do[rows])

    whole, alone = grads(slice(None)), grads(slice(9, 10))
    for i, (a, b) in enumerate(zip(alone, whole)):
        if i in (1, 3, 4):  # dk1, dk2, dv
            assert torch.equal(a[0], b[9])
