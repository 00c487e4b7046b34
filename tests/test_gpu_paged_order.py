"""Paged decode takes the (sequence, split) entries of a batch longest first when there is one thread per entry: every
sequence's result must be the one it has alone, bit for bit (the order changes no arithmetic)."""
import pytest
import torch

from flagattention_b200 import paged_attention
from gpu_util import device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,block", [(64, 16), (128, 32)])
@pytest.mark.parametrize("splits", [1, 2, 4])
@pytest.mark.parametrize("lens", [
    [1], [700, 700, 700],                       # nothing to order, nothing but ties
    [641 + i for i in range(12)], [640, 641, 640, 640, 640, 640],   # as many tiles each, one more in one of them
    [5, 1500, 128, 129, 1024, 1, 640],          # one key, edges of a 128-key tile, empty last splits
    [(37 * i) % 300 + 1 for i in range(192)],   # with two CTA splits as many entries as threads
    [(37 * i) % 900 + 1000 for i in range(192)],   # ... of blocks long enough to be ordered
    [(37 * i) % 300 + 1 for i in range(385)],   # more: the given order
])
def test_each_sequence_as_alone(lens, splits, D, block):
    g = torch.Generator(device=device()).manual_seed(len(lens))
    S, longest = len(lens), max(lens)
    Hkv = 32 if S < 100 else 2   # more blocks than SMs, or the order is left as given
    Hq = 4 * Hkv
    k, v = (torch.randn(64, Hkv, block, D, device=device(), dtype=torch.float16, generator=g) for _ in range(2))
    q = torch.randn(S, Hq, D, device=device(), dtype=torch.float16, generator=g)
    tables = torch.randint(0, 64, (S, -(-longest // block)), device=device(), dtype=torch.int32, generator=g)
    n = torch.tensor(lens, device=device(), dtype=torch.int32)
    got = paged_attention(q, k, v, n, tables, D ** -0.5, longest, splits)
    for i in sorted({0, 1 % S, S // 2, S - 1, lens.index(longest)}):
        alone = paged_attention(q[i:i + 1], k, v, n[i:i + 1], tables[i:i + 1], D ** -0.5, longest, splits)
        assert torch.equal(got[i:i + 1], alone), i
