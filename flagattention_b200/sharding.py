"""Multi-GPU partitioning of ``flash_attention`` without any collective.

The operator is independent per (batch, KV head): all query heads that share a KV head stay on one
rank, so dK/dV need no cross-rank reduction. ``unit_range`` assigns each rank a contiguous range
of the ``B * Hkv`` units; ``shard`` returns the matching views of q, k, v (and anything shaped
like q), one piece per batch the range touches. One process per GPU runs its pieces through the
ordinary ``flash_attention``.

Outputs are bit-identical to the corresponding slices of a single-GPU run, unless the piece has so few
query rows that the forward splits its keys (``split_kv.choose_num_splits``, which counts batch and heads).
So are dK and dV when the backward shares its key blocks between as many thread blocks for the piece as for
the whole (``b200attn_bwd_key_block_split`` of the C ABI tells; long sequences, more than 128 steps of 64
queries by the query heads of a KV head, never share): otherwise they agree to the order of fp32 sums before
one rounding. dQ at head dimensions 32 and up is summed in no fixed order by default; under
``torch.use_deterministic_algorithms(True)`` it is bit-identical like the outputs, given the same outputs.
"""
from __future__ import annotations

from typing import Iterator

import torch


def unit_range(num_units: int, rank: int, world: int) -> tuple[int, int]:
    """Contiguous, balanced split: the first ``num_units % world`` ranks get one extra unit."""
    if not 0 <= rank < world:
        raise ValueError(f"rank {rank} outside world of {world}")
    base, extra = divmod(num_units, world)
    start = rank * base + min(rank, extra)
    return start, start + base + (1 if rank < extra else 0)


def pieces(B: int, Hkv: int, rank: int, world: int) -> Iterator[tuple[int, int, int]]:
    """Yields ``(batch, kv_head_begin, kv_head_end)`` covering this rank's units."""
    lo, hi = unit_range(B * Hkv, rank, world)
    while lo < hi:
        b, h0 = divmod(lo, Hkv)
        h1 = min(Hkv, h0 + (hi - lo))
        yield b, h0, h1
        lo += h1 - h0


def shard(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, rank: int, world: int, *like_q: torch.Tensor):
    """List of ``(q_piece, k_piece, v_piece, *like_q_pieces)`` views owned by ``rank``."""
    B, Hq = q.shape[:2]
    Hkv = k.shape[1]
    groups = Hq // Hkv
    out = []
    for b, h0, h1 in pieces(B, Hkv, rank, world):
        qs = slice(h0 * groups, h1 * groups)
        out.append((q[b:b + 1, qs], k[b:b + 1, h0:h1], v[b:b + 1, h0:h1], *(t[b:b + 1, qs] for t in like_q)))
    return out
