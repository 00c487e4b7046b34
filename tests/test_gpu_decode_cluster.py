"""Decode over split keys: up to eight splits merge in a cluster, more through partial results and the combine kernel. Any
split count, with splits left empty by short or masked sequences, against the oracle, and the two ways against each other."""
import pytest
import torch

from flagattention_b200 import _lib
from gpu_util import assert_2x_rule, attention_forward, device, make_qkv

pytestmark = pytest.mark.gpu


def _decode(q, k, v, causal, splits):
    B, Hq, M, D = q.shape
    o, lse = torch.full_like(q, float("nan")), torch.full((B, Hq, M), float("nan"), device=device())
    part = torch.empty(B * Hq * M * splits * (D + 1), device=device())
    p = _lib.SplitKVParams(_lib.tensor4(q), _lib.tensor4(k), _lib.tensor4(v), _lib.tensor4(o), lse.data_ptr(), part.data_ptr(),
                           part.data_ptr() + 4 * B * Hq * M * splits * D, B, Hq, k.shape[1], M, k.shape[2], D, splits,
                           _lib.dtype_code(q.dtype), int(causal), D ** -0.5, None)
    _lib.check(_lib.load().b200attn_fwd_splitkv(p, torch.cuda.current_stream().cuda_stream), "b200attn_fwd_splitkv")
    return o, lse


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [16, 64, 128])
@pytest.mark.parametrize("G,M,N,causal", [(1, 1, 1, False), (1, 1, 129, False), (2, 1, 3000, False), (1, 2, 1025, True), (1, 2, 1, True)])
def test_split_counts(G, M, N, causal, D, dtype):
    q, k, v, _ = make_qkv(2, 3 * G, 3, M, N, D, dtype, seed=N)
    ref, l_ref, _ = attention_forward(q, k, v, causal, upcast=True, return_log_normalizer=True)
    low = attention_forward(q, k, v, causal, upcast=False)
    seen = torch.isfinite(l_ref)
    for splits in (1, 2, 3, 7, 8, 9, 16):
        o, lse = _decode(q, k, v, causal, splits)
        assert_2x_rule(f"{splits} splits", o, low, ref, slack=2e-5)
        assert torch.equal(torch.isfinite(lse), seen) and (lse - l_ref)[seen].abs().le(1e-4).all()
