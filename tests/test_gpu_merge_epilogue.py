"""The forward that combines its rows with a partial result over other keys against two partial results merged by their
own kernel: the same fp32 arithmetic, hence the same 16-bit rows up to a neighbouring number where the compiler
contracts differently."""
import pytest
import torch

from flagattention_b200 import _lib, piecewise, piecewise_attention
from gpu_util import device, make_qkv

pytestmark = pytest.mark.gpu


def _run(q, k, v, out, lse, band, partial=None):
    B, Hq, M, D = q.shape
    p = _lib.FwdParams(_lib.tensor4(q), _lib.tensor4(k), _lib.tensor4(v), _lib.tensor4(out), lse.data_ptr(), B, Hq, k.shape[1], M,
                       k.shape[2], D, _lib.dtype_code(q.dtype), _lib.dtype_code(out.dtype), 0, D ** -0.5, 0.0, 0, 0, None, 1, *band)
    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    if partial is None:
        _lib.check(lib.b200attn_fwd(p, stream), "b200attn_fwd")
    else:
        _lib.check(lib.b200attn_fwd_merge(p, partial[0].data_ptr(), partial[1].data_ptr(), stream), "b200attn_fwd_merge")


@pytest.mark.parametrize("layout", ["BHTD", "BTHD"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [16, 32, 64, 128])
@pytest.mark.parametrize("M,N,near,far", [
    (1, 1, (0, 1), (1, 2 ** 31 - 1)),                    # the far region is empty
    (127, 127, (0, 64), (64, 2 ** 31 - 1)),              # empty for the first rows, an edge inside a tile
    (257, 300, (0, 10), (128, 2 ** 31 - 1)),             # rows with nothing in either are none, a gap between
    (129, 65, (5, 6), (-2 ** 31, 5)),                    # the open side, rows without any key
    (200, 200, (1000, 1001), (-2 ** 31, 5000)),          # nothing near, no limit within reach far
    (200, 200, (1000, 1001), (-2 ** 31, 2 ** 31 - 1)),   # ... and none at all
])
def test_against_the_merge_kernel(M, N, near, far, D, dtype, layout):
    q, k, v, _ = make_qkv(2, 3, 3, M, N, D, dtype, layout=layout, seed=M)
    o_a, o_b = (torch.empty(2, 3, M, D, device=device()) for _ in range(2))
    l_a, l_b, l_got = (torch.empty(2, 3, M, device=device()) for _ in range(3))
    _run(q, k, v, o_a, l_a, near)
    _run(q, k, v, o_b, l_b, far)
    got, want = torch.empty_like(q), torch.empty_like(q)
    _run(q, k, v, got, l_got, far, (o_a, l_a))
    _lib.check(_lib.load().b200attn_merge_partial_store(
        o_a.data_ptr(), l_a.data_ptr(), o_b.data_ptr(), l_b.data_ptr(), 2, 3, M, D, _lib.tensor4(want),
        _lib.dtype_code(dtype), torch.cuda.current_stream().cuda_stream), "merge_partial_store")
    assert torch.equal(torch.isfinite(l_got), torch.isfinite(l_a))
    seen = torch.isfinite(l_a)
    assert (l_got - l_a)[seen].abs().le(1e-6 * (1 + l_a[seen].abs())).all()
    ulp = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10
    # Without any limit the two D = 128 launches take different pipelines, whose running maxima scale P differently before
    # it is rounded to 16 bits: half an ulp of P on each side, times the largest |v|.
    slack = ulp * v.float().abs().max() if far[1] == 2 ** 31 - 1 and far[0] == -2 ** 31 else 1e-6
    assert (got.float() - want.float()).abs().le(ulp * want.float().abs() + slack).all()


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_both_ways_of_the_operator(D, causal, monkeypatch):
    """More work items than SMs, where head dimensions up to 64 merge in a kernel of their own."""
    inputs = [torch.randn(3, 50, 257, D, device=device(), dtype=torch.float16, generator=torch.Generator(device()).manual_seed(i))
              for i in range(5)]
    assert piecewise._merges_in_epilogue(150, 257, D, 148) == (D == 128) and piecewise._merges_in_epilogue(74, 257, D, 148)
    got = {}
    for epilogue in (False, True):
        monkeypatch.setattr(piecewise, "_merges_in_epilogue", lambda *args: epilogue)
        leaves = [t.clone().requires_grad_() for t in inputs]
        o = piecewise_attention(*leaves, 100, causal=causal)
        got[epilogue] = (o.detach(),) + torch.autograd.grad(o, leaves[4], inputs[0])
    for a, b in zip(got[False], got[True]):   # neighbouring fp16 numbers where the compiler contracts differently
        a, b = a.float(), b.float()
        assert (a - b).abs().le(2.0 ** -10 * b.abs() + 1e-4 * b.abs().max()).all()
