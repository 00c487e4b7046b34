"""The dK/dV pass with several blocks per key block (a cluster that sums in shared memory) against the pass with one:
a (batch, KV head) pair by itself takes the first, the same pair among many the second. Both sum the same fp32 terms, in
another order, before one rounding to 16 bits."""
import pytest
import torch

from flagattention_b200 import flash_attention, piecewise_attention
from gpu_util import make_qkv

pytestmark = pytest.mark.gpu

# Values that differ by the order of fp32 sums round to the same or to neighbouring 16-bit numbers; neighbours just
# above a power of two are 2^-7 (bf16, 7 stored bits) and 2^-10 (fp16) of the value apart.
_REL = {torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10}


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
