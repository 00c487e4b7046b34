"""The dK/dV pass with several blocks per key block (a cluster that sums in shared memory) against the pass with one:
a (batch, KV head) pair by itself takes the first, the same pair among many the second. Both sum the same fp32 terms, in
another order, before one rounding to 16 bits."""
import pytest
import torch

from flagattention_b200 import _lib, flash_attention, piecewise_attention
from flagattention_b200.sharding import shard
from gpu_util import assert_2x_rule, attention_backward, attention_forward, kernel_dropout_mask, make_qkv

pytestmark = pytest.mark.gpu

# Values that differ by the order of fp32 sums round to the same or to neighbouring 16-bit numbers; neighbours just
# above a power of two are 2^-7 (bf16, 7 stored bits) and 2^-10 (fp16) of the value apart.
_REL = {torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10}


def _shared(*call):
    return _lib.load().b200attn_bwd_key_block_split(*map(int, call))


def _close(a, b, name=''):
    tol = _REL[a.dtype]
    a, b = a.float(), b.float()
    # (1e-4 of the largest element: what fp32 sums of up to 2048 terms lose where they cancel)
    diff, bound = (a - b).abs(), tol * torch.maximum(a.abs(), b.abs()) + 1e-4 * b.abs().max()
    bad = int((diff / bound).argmax())
    assert (diff <= bound).all(), (name, int((diff > bound).sum()), diff.numel(), bad, a.flatten()[bad].item(), b.flatten()[bad].item(), b.abs().max().item())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("G,M,N,causal", [
    (8, 512, 512, True),      # whole heads per block
    (1, 2000, 130, False),    # one head split between blocks, two keys in the last key block
    (24, 65, 129, True),      # two steps per head, one key in the last key block
    (12, 200, 1025, True),    # more keys than queries
])
# (enough query rows that no forward takes the split-key branch, whose outputs round differently)
def test_pair_alone_equals_pair_among_many(G, M, N, D, causal, dtype):
    q, k, v, do = make_qkv(1, G, 1, M, N, D, dtype, seed=5, requires_grad=True)
    alone = torch.autograd.grad(flash_attention(q, k, v, causal), (q, k, v), do)
    many = -(-8 * 160 // -(-N // 128))   # more key blocks than four times any number of resident blocks
    assert _shared(1, G, 1, M, N, D, causal) > 1 and _shared(many, G, 1, M, N, D, causal) == 1
    big = [t.detach().expand(many, -1, -1, -1).contiguous().requires_grad_() for t in (q, k, v)]
    grads = torch.autograd.grad(flash_attention(*big, causal), big, do.expand(many, -1, -1, -1).contiguous())
    for name, a, b in zip(("dq", "dk", "dv"), alone, grads):
        _close(a[0], b[-1], name)


def test_added_gradient_of_the_second_region():
    """Piecewise attention adds the far region's dV onto the near region's in the pass itself."""
    inputs = [torch.randn(1, 2, 700, 64, device="cuda", dtype=torch.bfloat16) for _ in range(5)]
    do = torch.randn_like(inputs[0])
    leaves = [t.clone().requires_grad_() for t in inputs]
    alone = torch.autograd.grad(piecewise_attention(*leaves, 256, causal=True), leaves, do)
    big = [t.expand(128, -1, -1, -1).contiguous().requires_grad_() for t in inputs]
    grads = torch.autograd.grad(piecewise_attention(*big, 256, causal=True), big, do.expand(128, -1, -1, -1).contiguous())
    for a, b in zip(alone, grads):
        # (dV is rounded twice here: after each region)
        af, bf = a[0].float(), b[-1].float()
        assert (af - bf).abs().le(2.0 ** -6 * torch.maximum(af.abs(), bf.abs()) + 2.0 ** -8 * bf.abs().max()).all()


# (number of blocks per key block, call): every number that the rule can give
_COUNTS = [(2, (8, 8, 2, 1024, 1024, 128)), (4, (4, 8, 2, 1024, 1024, 128)), (8, (4, 4, 1, 1024, 1024, 64)), (8, (1, 8, 1, 512, 512, 128)), (8, (1, 8, 1, 512, 512, 64)),
           (4, (1, 8, 1, 512, 512, 32)), (2, (1, 8, 1, 512, 512, 16)), (8, (1, 2, 2, 1000, 700, 128))]


def _check_against_oracle(q, k, v, do, causal, grads, p=0.0, mask=None):
    ref = attention_backward(q.detach(), k.detach(), v.detach(), do, causal, dropout_p=p, dropout_mask=mask)
    leaves = [t.detach().clone().requires_grad_() for t in (q, k, v)]
    low = torch.autograd.grad(attention_forward(*leaves, causal, dropout_p=p, dropout_mask=mask, upcast=False), leaves, do)
    for name, a, b, c in zip(("dq", "dk", "dv"), grads, low, ref):
        assert_2x_rule(name, a, b, c)


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("count,call", _COUNTS)
def test_every_count_against_the_oracle(count, call, deterministic):
    B, Hq, Hkv, M, N, D = call
    assert _shared(*call, True) == count
    q, k, v, do = make_qkv(B, Hq, Hkv, M, N, D, torch.bfloat16, seed=9, requires_grad=True)
    torch.use_deterministic_algorithms(deterministic)
    try:
        grads = torch.autograd.grad(flash_attention(q, k, v, True), (q, k, v), do)
    finally:
        torch.use_deterministic_algorithms(False)
    _check_against_oracle(q, k, v, do, True, grads)


@pytest.mark.parametrize("G,M,N,D,causal", [
    (8, 512, 512, 128, True), (8, 512, 512, 64, True), (4, 600, 200, 32, False), (8, 512, 512, 16, True),
    (1, 2000, 130, 64, False),   # the share begins inside a head
])
def test_dropout_in_shared_key_blocks(G, M, N, D, causal):
    """A share's keep words and its head, the scale of dV after the exchange."""
    assert _shared(1, G, 1, M, N, D, causal) > 1
    q, k, v, do = make_qkv(1, G, 1, M, N, D, torch.float16, seed=2, requires_grad=True)
    torch.cuda.manual_seed(3)
    o, _, _, seed, offset = flash_attention(q, k, v, causal, dropout_p=0.2, return_seed_offset=True)
    grads = torch.autograd.grad(o, (q, k, v), do)
    _check_against_oracle(q, k, v, do, causal, grads, 0.2, kernel_dropout_mask(1, G, M, N, 0.2, seed, offset))


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("B,Hq,Hkv,M,N,D,causal", [
    (4, 8, 1, 2048, 2048, 128, True),    # more than 128 steps: never shared
    (2, 16, 4, 2500, 2500, 64, True),
    (2, 8, 2, 512, 512, 128, True),      # eight blocks for the whole and for each batch
    (4, 64, 1, 512, 512, 64, True),      # more than 128 steps by the heads of one KV head
])
def test_pieces_with_the_same_count_give_the_bits_of_the_whole(B, Hq, Hkv, M, N, D, causal, deterministic):
    q, k, v, do = make_qkv(B, Hq, Hkv, M, N, D, torch.bfloat16, seed=5)

    def grads(q, k, v, do):
        leaves = [t.detach().requires_grad_() for t in (q, k, v)]
        o = flash_attention(*leaves, causal)
        return (o.detach(),) + torch.autograd.grad(o, leaves, do)

    compared = 0
    torch.use_deterministic_algorithms(deterministic)
    try:
        o, dq, dk, dv = grads(q, k, v, do)
        for rank in range(4):
            for (qp, kp, vp, dop), (op, dkp, dvp, dqp) in zip(shard(q, k, v, rank, 4, do), shard(o, dk, dv, rank, 4, dq)):
                if _shared(*qp.shape[:2], kp.shape[1], M, N, D, causal) != _shared(B, Hq, Hkv, M, N, D, causal):
                    continue
                got = grads(qp, kp, vp, dop)
                assert torch.equal(got[0], op) and torch.equal(got[2], dkp) and torch.equal(got[3], dvp)
                assert not deterministic or torch.equal(got[1], dqp)
                compared += 1
    finally:
        torch.use_deterministic_algorithms(False)
    assert compared
