"""The native host path against the Python one it stands in front of: same results for every form that it takes, and every
other form handed on (copies, wrong arguments, transforms)."""
import sys
import threading
import time

import pytest
import torch

from flagattention_b200 import _lib, flash_attention, flash_attention_split_kv, paged_attention, status
from gpu_util import device, make_qkv

pytestmark = pytest.mark.gpu


class _Declines:
    """A host path that takes nothing: every call runs in Python."""

    def __getattr__(self, name):
        return lambda *args: None


def _native(o):
    """Whether the result's backward is the C++ node."""
    return "FlashAttentionFunction" not in o.grad_fn.name()


def _both(monkeypatch, call):
    _lib.host()
    native = call()
    with monkeypatch.context() as m:
        m.setattr(_lib, "_HOST", _Declines())
        return native, call()


@pytest.mark.parametrize("layout", ["BHTD", "BTHD"])
@pytest.mark.parametrize("B,Hq,Hk,M,N,D,dtype", [
    (1, 4, 4, 128, 128, 64, torch.float16), (2, 6, 2, 77, 201, 128, torch.bfloat16), (1, 2, 1, 1, 3000, 64, torch.float16),
    (1, 8, 2, 3, 5000, 128, torch.bfloat16), (3, 16, 16, 300, 1, 32, torch.float16)])
def test_same_results(B, Hq, Hk, M, N, D, dtype, layout, monkeypatch):
    q, k, v, do = make_qkv(B, Hq, Hk, M, N, D, dtype, layout=layout, seed=4, requires_grad=True)
    torch.use_deterministic_algorithms(True)  # (dQ bit for bit)
    try:
        def train():
            o = flash_attention(q, k, v, causal=True, sm_scale=0.2)
            assert _native(o) != isinstance(_lib.host(), _Declines)
            return (o.detach(),) + torch.autograd.grad(o, (q, k, v), do)
        a, b = _both(monkeypatch, train)
    finally:
        torch.use_deterministic_algorithms(False)
    for x, y in zip(a, b):
        assert torch.equal(x, y) and x.stride() == y.stride()
    x, y = _both(monkeypatch, lambda: flash_attention_split_kv(q, k, v))
    assert torch.equal(x, y) and not x.requires_grad


def test_same_paged_results(monkeypatch):
    g = torch.Generator(device=device()).manual_seed(0)
    q = torch.randn(3, 8, 64, device=device(), dtype=torch.float16, generator=g)
    k, v = (torch.randn(40, 2, 16, 64, device=device(), dtype=torch.float16, generator=g) for _ in range(2))
    lens = torch.tensor([200, 1, 77], device=device(), dtype=torch.int32)
    tables = torch.randint(0, 40, (3, 13), device=device(), dtype=torch.int32, generator=g)
    for lens_, tables_, splits in ((lens, tables, 0), (lens, tables, 3), (lens.long(), tables, 0), (lens, tables.long(), 2)):
        x, y = _both(monkeypatch, lambda: paged_attention(q, k, v, lens_, tables_, 0.125, 200, splits))
        assert torch.equal(x, y)


def test_forms_that_are_handed_on():
    host = _lib.host()
    q, k, v, _ = make_qkv(2, 4, 2, 64, 64, 64, torch.float16, seed=1)
    assert host.flash(q, k, v, False, None) is not None
    odd = torch.randn(2, 4, 64, 65, device=device(), dtype=torch.float16)[..., 1:]      # rows off 16 bytes
    wide = torch.randn(2, 4, 64, 128, device=device(), dtype=torch.float16)[..., ::2]   # feature stride 2
    for bad in ((odd, k, v), (wide, k, v), (q.cpu(), k, v), (q.float(), k.float(), v.float()), (q, k.bfloat16(), v), (q[0], k[0], v[0]),
                (q, k[:, :, :32], v), (q[:1], k, v), (q[:, :3], k, v), (q[..., :48], k[..., :48], v[..., :48]), (q, k, None)):
        assert host.flash(*bad, False, None) is None and host.split_kv(*bad, False, None) is None
    ref = flash_attention(wide.contiguous(), k, v)
    assert torch.equal(flash_attention(wide, k, v), ref)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda x: flash_attention(x, x, x))(torch.stack([q, q]))
    with pytest.raises(AssertionError):
        flash_attention(q[:, :3], k, v)


class _Named(torch.Tensor):
    """A subclass without __torch_dispatch__, whose operations return it again."""


def test_subclasses_come_back_as_from_python(monkeypatch):
    q, k, v, _ = make_qkv(2, 4, 2, 64, 64, 64, torch.float16, seed=2)
    named = q.as_subclass(_Named)
    x, y = _both(monkeypatch, lambda: flash_attention(named, k, v))
    assert type(x) is type(y) is _Named and torch.equal(x.as_subclass(torch.Tensor), flash_attention(q, k, v))
    host = _lib.host()
    assert host.flash(named, k, v, False, None) is None and host.split_kv(q, k.as_subclass(_Named), v, False, None) is None
    assert host.flash(torch.nn.Parameter(q), k, v, False, None) is not None


def test_calls_are_taken_after_a_transform_and_a_compilation():
    """(also what makes the tests below, and in the files behind this one, run the native path)"""
    host = _lib.host()
    q, k, v, _ = make_qkv(2, 4, 2, 64, 64, 64, torch.float16, seed=1)
    lens, tables = torch.tensor([40, 64], device=device(), dtype=torch.int32), torch.zeros(2, 4, device=device(), dtype=torch.int32)
    cache = torch.randn(3, 2, 16, 64, device=device(), dtype=torch.float16)

    def taken():
        return [x is not None for x in (host.flash(q, k, v, False, None), host.split_kv(q, k, v, False, None),
                                        host.paged(q[:, :, 0].contiguous(), cache, cache, lens, tables, 0.125, 64, 0))]
    torch.func.vmap(lambda x: x + 1)(q)
    assert taken() == [True] * 3
    torch.compile(lambda x: x * 2 + 1, backend="eager")(q)
    assert taken() == [True] * 3


def test_gradient_of_another_type_stride_and_only_some_inputs():
    q, k, v, do = make_qkv(1, 4, 4, 160, 160, 64, torch.float16, seed=3)
    k.requires_grad_()
    o = flash_attention(q, k, v)
    assert _native(o)
    a, = torch.autograd.grad(o, k, do, retain_graph=True)
    b, = torch.autograd.grad(o, k, do.transpose(1, 2).contiguous().transpose(1, 2), retain_graph=True)
    assert torch.equal(a, b)
    c, = torch.autograd.grad(o.float().sum(), k)        # an expanded gradient
    d, = torch.autograd.grad(flash_attention(q, k, v), k, torch.ones_like(o))
    assert torch.equal(c, d)


@pytest.mark.parametrize("call", ["flash", "split_kv", "paged"])
def test_other_threads_run_while_a_call_waits(call, monkeypatch):
    """A call that has to wait for room in the launch queue does not hold the GIL. With a switch interval far beyond the
    test's length another thread gets it only from a call that lets go of it (the status poll, which would, is put off)."""
    q, k, v, _ = make_qkv(2, 4, 2, 64, 64, 64, torch.float16, seed=1)
    q1 = q[:, :, 0].contiguous()
    lens, tables = torch.tensor([40, 64], device=device(), dtype=torch.int32), torch.zeros(2, 4, device=device(), dtype=torch.int32)
    cache = torch.randn(3, 2, 16, 64, device=device(), dtype=torch.float16)
    host = _lib.host()
    run = {"flash": lambda: host.flash(q, k, v, False, None), "split_kv": lambda: host.split_kv(q, k, v, False, None),
           "paged": lambda: host.paged(q1, cache, cache, lens, tables, 0.125, 64, 0)}[call]
    assert run() is not None
    status.check_device_status(device())
    monkeypatch.setattr(status, "POLL_INTERVAL_S", float("inf"))
    turns, stop = [0], threading.Event()

    def other():
        while not stop.is_set():
            turns[0] += 1
            time.sleep(0.001)
    interval = sys.getswitchinterval()
    thread = threading.Thread(target=other)
    sys.setswitchinterval(1000.0)
    try:
        thread.start()
        torch.cuda._sleep(int(3e8))   # about 0.15 s on the device, in which the queue fills up
        before = turns[0]
        for _ in range(3000):
            run()
        got = turns[0] - before
    finally:
        stop.set()
        sys.setswitchinterval(interval)
        thread.join()
        torch.cuda.synchronize()
    assert got > 10


def test_saved_tensor_hooks_see_what_is_kept():
    q, k, v, do = make_qkv(1, 2, 2, 256, 256, 64, torch.float16, seed=6, requires_grad=True)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.cpu(), lambda t: t.to(device())):
        o = flash_attention(q, k, v)
    assert _native(o) and len(packed) >= 4
    ref = torch.autograd.grad(flash_attention(q, k, v), (k, v), do)
    for x, y in zip(torch.autograd.grad(o, (k, v), do), ref):
        assert torch.equal(x, y)
