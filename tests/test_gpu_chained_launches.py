"""Decode launches follow one another so closely that a kernel is resident while its predecessor still runs. A chain of
small steps over one scratch buffer, each with inputs of its own, must give what the steps give one by one."""
import pytest
import torch

from flagattention_b200 import _lib
from gpu_util import device, make_qkv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hq,Hkv,N,D,splits", [
    (2, 4, 4, 1500, 64, 12),    # streaming kernel, combine kernel
    (2, 8, 2, 1500, 128, 6),    # tensor-core kernel, combine kernel
    (3, 4, 4, 600, 128, 5),     # streaming kernel, merged in a cluster
])
def test_chain_equals_single_steps(B, Hq, Hkv, N, D, splits):
    lib, steps = _lib.load(), 24
    inputs = [make_qkv(B, Hq, Hkv, 1, N, D, torch.float16, seed=i)[:3] for i in range(steps)]
    part = torch.empty(B * Hq * splits * (D + 1), device=device())
    lse = torch.empty(B, Hq, 1, device=device())

    def step(i, out):
        q, k, v = inputs[i]
        p = _lib.SplitKVParams(_lib.tensor4(q), _lib.tensor4(k), _lib.tensor4(v), _lib.tensor4(out), lse.data_ptr(), part.data_ptr(),
                               part.data_ptr() + 4 * B * Hq * splits * D, B, Hq, Hkv, 1, N, D, splits, _lib.dtype_code(q.dtype), 0,
                               D ** -0.5, None)
        _lib.check(lib.b200attn_fwd_splitkv(p, torch.cuda.current_stream().cuda_stream), "b200attn_fwd_splitkv")

    want = [torch.empty_like(x[0]) for x in inputs]
    for i in range(steps):
        step(i, want[i])
        torch.cuda.synchronize()
    got = [torch.empty_like(x[0]) for x in inputs]
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        for i in range(steps):
            step(i, got[i])
    for _ in range(20):
        for t in got:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("B,H,N,D,splits", [(2, 4, 1500, 64, 12), (3, 4, 600, 128, 5)])
def test_result_as_the_next_query(B, H, N, D, splits):
    lib, steps = _lib.load(), 24
    q, k, v, _ = make_qkv(B, H, H, 1, N, D, torch.float16, seed=1)
    part = torch.empty(B * H * splits * (D + 1), device=device())
    lse = torch.empty(B, H, 1, device=device())
    ring = [q.clone(), torch.empty_like(q)]

    def run(wait):
        ring[0].copy_(q)
        for i in range(steps):
            a, o = ring[i % 2], ring[1 - i % 2]
            p = _lib.SplitKVParams(_lib.tensor4(a), _lib.tensor4(k), _lib.tensor4(v), _lib.tensor4(o), lse.data_ptr(), part.data_ptr(),
                                   part.data_ptr() + 4 * B * H * splits * D, B, H, H, 1, N, D, splits, _lib.dtype_code(q.dtype), 0,
                                   4.0, None)
            _lib.check(lib.b200attn_fwd_splitkv(p, torch.cuda.current_stream().cuda_stream), "b200attn_fwd_splitkv")
            if wait:
                torch.cuda.synchronize()
        return ring[steps % 2].clone()

    want = run(True)
    for _ in range(20):
        assert torch.equal(run(False), want)
