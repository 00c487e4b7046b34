"""The forward with one query tile per block (16-bit outputs, head dimensions up to 64) at the edges of its tiles: rows
around 128, keys around the 64 of a step, single rows and keys, far band edges, dropout drawn and read from the cache."""
import pytest
import torch

from flagattention_b200 import _lib, flash_attention
from flagattention_b200 import flash as flash_mod
from gpu_util import assert_2x_rule, attention_forward, device, kernel_dropout_mask, make_qkv, max_abs_diff

pytestmark = pytest.mark.gpu


def _forward(q, k, v, causal=False, band=None):
    """Straight through the C ABI, so that no shape takes the split-key branch."""
    B, Hq, M, D = q.shape
    o = torch.full_like(q, float("nan"))
    lse = torch.full((B, Hq, M), float("nan"), device=q.device)
    dt = _lib.dtype_code(q.dtype)
    p = _lib.FwdParams(_lib.tensor4(q), _lib.tensor4(k), _lib.tensor4(v), _lib.tensor4(o), lse.data_ptr(), B, Hq, k.shape[1], M,
                       k.shape[2], D, dt, dt, int(causal), D ** -0.5, 0.0, 0, 0, None, int(band is not None), *(band or (0, 0)))
    _lib.check(_lib.load().b200attn_fwd(p, torch.cuda.current_stream().cuda_stream), "b200attn_fwd")
    return o, lse


@pytest.mark.parametrize("layout", ["BHTD", "BTHD"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("M,N,causal", [(1, 1, False), (127, 63, False), (128, 64, True), (129, 65, True), (257, 320, True),
                                        (300, 100, True), (64, 1000, False)])
def test_tile_edges(M, N, causal, D, dtype, layout):
    q, k, v, _ = make_qkv(2, 4, 2, M, N, D, dtype, layout=layout, seed=M + N)
    o, lse = _forward(q, k, v, causal)
    ref, l_ref, _ = attention_forward(q, k, v, causal, upcast=True, return_log_normalizer=True)
    assert_2x_rule("o", o, attention_forward(q, k, v, causal, upcast=False), ref)
    seen = torch.isfinite(l_ref)
    assert torch.equal(seen, torch.isfinite(lse)) and max_abs_diff(lse[seen], l_ref[seen]) <= 1e-4


@pytest.mark.parametrize("D", [32, 64])
@pytest.mark.parametrize("M,N,band", [(200, 200, (0, 70)), (130, 500, (-40, 64)), (129, 129, (100, 2 ** 31 - 1))])
def test_band_edges(M, N, band, D):
    q, k, v, _ = make_qkv(1, 2, 2, M, N, D, torch.float16, seed=1)
    o, lse = _forward(q, k, v, band=band)
    s = (q.float() @ k.float().transpose(-1, -2)) * D ** -0.5
    d = torch.arange(M, device=device())[:, None] + (N - M) - torch.arange(N, device=device())
    s = s.masked_fill(~((d >= band[0]) & (d < band[1])), float("-inf"))
    l_ref = torch.logsumexp(s, -1)
    ref = torch.nan_to_num(torch.softmax(s, -1)) @ v.float()
    seen = torch.isfinite(l_ref)
    assert torch.equal(seen, torch.isfinite(lse)) and (lse[seen] - l_ref[seen]).abs().max() <= 1e-4
    # P and the result are rounded to 11 bits: |v| < 5 here
    assert (o.float() - ref).abs().max() <= 5 * 2.0 ** -10


@pytest.mark.parametrize("limit", [0, 1 << 30])  # decisions drawn in the forward, read from the cache
@pytest.mark.parametrize("M,N,causal", [(1900, 65, False), (2000, 193, True)])
def test_dropout(M, N, causal, limit, monkeypatch):
    monkeypatch.setattr(flash_mod, "_KEEP_MASK_LIMIT", limit)
    q, k, v, _ = make_qkv(1, 2, 1, M, N, 64, torch.float16, seed=2, requires_grad=True)
    torch.cuda.manual_seed(11)
    o, _, _, seed, offset = flash_attention(q, k, v, causal, dropout_p=0.3, return_seed_offset=True)
    keep = kernel_dropout_mask(1, 2, M, N, 0.3, seed, offset)
    ref = attention_forward(q, k, v, causal, dropout_p=0.3, dropout_mask=keep, upcast=True)
    low = attention_forward(q, k, v, causal, dropout_p=0.3, dropout_mask=keep, upcast=False)
    assert_2x_rule("o", o.detach(), low.detach(), ref.detach())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("N,causal", [(128, False), (128, True), (97, False)])
def test_error_of_short_rows_is_that_of_exact_maxima(N, causal, D, dtype):
    """Rows of up to 128 keys: the largest probability of a row is 1 and takes no rounding error. The error of O in the
    2-norm (over 5e5 and more elements) is at most that of the model with P rounded against each row's own maximum, and
    a hundredth for the approximation of exp2 and the model's rounding of its first half (P rounded against the maximum
    of the first 64 keys alone is 2 % and more above it)."""
    q, k, v, _ = make_qkv(4, 64, 64, 128, N, D, dtype, seed=N)
    o, _ = _forward(q, k, v, causal)
    s = (q.double() @ k.double().transpose(-1, -2)) * D ** -0.5
    if causal:
        hidden = torch.arange(N, device=device()) > torch.arange(128, device=device())[:, None] + (N - 128)
        s = s.masked_fill(hidden, float("-inf"))
    p = torch.exp(s - s.amax(-1, keepdim=True))
    exact = (p @ v.double()) / p.sum(-1, keepdim=True)
    model = ((p.to(dtype).double() @ v.double()) / p.sum(-1, keepdim=True)).to(dtype).double()
    assert (o.double() - exact).norm() <= 1.01 * (model - exact).norm()
