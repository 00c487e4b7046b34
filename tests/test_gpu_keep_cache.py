"""The kernel that draws the dropout decisions into the cache against the draws inside the forward and backward
kernels: the same decisions, hence (separate backward kernels) the same results bit for bit."""
import pytest
import torch

from flagattention_b200 import flash as flash_mod
from flagattention_b200 import flash_attention
from gpu_util import make_qkv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,M,N,D,causal,offset", [
    (1, 2, 257, 33, 64, False, 0),                  # one row in the second row block, one key in the second word
    (1, 3, 128, 129, 128, True, (1 << 32) - 8000),  # the counter's low word wraps inside a run of 32
    (1, 2, 513, 640, 32, True, (1 << 31) - 40),     # 32-bit counters that run past 2^31
    (70000, 1, 16, 16, 16, True, 1 << 33),          # more heads than the grid's second dimension holds
    (2, 3, 640, 1, 128, False, 0),                  # the dQ pass: one word, none behind it for the step's second half
    (2, 3, 640, 90, 64, False, 0),                  # ... three words, the fourth is the next head's
    (2, 3, 640, 97, 16, True, 0),                   # ... and four, one key in the last
])
def test_cached_decisions_equal_drawn_decisions(B, H, M, N, D, causal, offset, monkeypatch):
    q, k, v, do = make_qkv(B, H, H, M, N, D, torch.float16, seed=3, requires_grad=True)
    if B * H * M < 16 * 148:  # enough rows that the call does not take the split-key branch, which has no dropout
        q, k, v, do = (t.repeat(64, 1, 1, 1).detach() for t in (q, k, v, do))
        q, k, v = (t.requires_grad_() for t in (q, k, v))
    generator = torch.cuda.default_generators[0]

    def results(limit):
        monkeypatch.setattr(flash_mod, "_KEEP_MASK_LIMIT", limit)
        torch.cuda.manual_seed(99)
        state = generator.get_state()
        state.view(torch.int64)[1] = offset
        generator.set_state(state)
        torch.use_deterministic_algorithms(True)
        try:
            o = flash_attention(q, k, v, causal, dropout_p=0.25)
            return (o,) + torch.autograd.grad(o, (q, k, v), do)
        finally:
            torch.use_deterministic_algorithms(False)

    for cached, drawn in zip(results(1 << 30), results(0)):
        assert torch.equal(cached, drawn)
