"""The native host path's copy of the split-KV rule against the Python one, that it takes no CPU tensor, and in which
modes of torch it takes calls."""
import random

import torch
from torch._subclasses import FakeTensorMode

from flagattention_b200 import _lib
from flagattention_b200.split_kv import choose_num_splits


def test_split_rule_agrees():
    rnd = random.Random(0)
    host = _lib.host()
    shapes = [(b, h, m, n) for b in (1, 2, 9) for h in (1, 8, 118, 119) for m in (1, 16, 17) for n in (1, 128, 129, 4096, 100000)]
    shapes += [(rnd.randint(1, 8), rnd.randint(1, 40), rnd.randint(1, 300), rnd.randint(1, 40000)) for _ in range(3000)]
    for s in shapes:
        for sms in (148, 132, 1):
            assert host.takes_split_branch(*s, sms) == (choose_num_splits(*s, sms) > 1), (s, sms)


def test_cpu_tensors_are_handed_on():
    q = torch.randn(1, 2, 16, 64)
    host = _lib.host()
    assert host.flash(q, q, q, False, None) is None and host.split_kv(q, q, q, False, None) is None
    assert host.paged(q[0], q, q, torch.ones(2, dtype=torch.int32), torch.zeros(2, 1, dtype=torch.int32), 0.1, 4, 0) is None


def test_ordinary_mode_ends_and_comes_back():
    """Transforms, dispatch modes and tracers are handed on while they are active, and not for the rest of the thread."""
    ordinary = _lib.host().ordinary_mode
    x = torch.ones(3)
    seen = []

    def look(t):
        seen.append(ordinary())
        return t * 2

    assert ordinary()
    torch.func.vmap(look)(x)
    torch.func.grad(lambda t: look(t).sum())(x)
    torch.func.jvp(look, (x,), (x,))
    torch.func.vmap(torch.func.grad(lambda t: look(t).sum()))(torch.ones(2, 3))
    torch.func.functionalize(look)(x)
    assert seen == [False] * 5 and ordinary()
    with FakeTensorMode():
        assert not ordinary()
    torch.jit.trace(look, x, check_trace=False)
    assert seen[5:] == [False] and ordinary()
    torch.compile(lambda t: t * 2 + 1, backend="eager")(x)
    assert ordinary()
