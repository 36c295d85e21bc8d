"""Branches of a captured step (`ops/branch.py`): they share no scratch memory with what runs beside them."""

from __future__ import annotations

import gc
import sys
import threading
from types import SimpleNamespace

import pytest
import torch

from semantic_aware_adaptive_kv_cache_precision_b200 import ops
from semantic_aware_adaptive_kv_cache_precision_b200.ops import _lib, branch
from semantic_aware_adaptive_kv_cache_precision_b200.ops.branch import apart

DEV = "cuda"
STEP = SimpleNamespace(is_decode=True)


def captured(run):
    """`run()` in a graph, after one run outside; (graph, the captured run's result)."""
    run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run()
    return graph, out


def attention_case(dim, seed, keys=700, tokens=2, heads=2):
    """A decoded token of each of two sequences over caches in blocks, its keys shared out over four blocks."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    blocks = -(-keys // ops.CACHE_BLOCK)
    cache = [torch.randn((tokens * blocks, heads, ops.CACHE_BLOCK, dim), generator=g, device=DEV).bfloat16()
             for _ in range(2)]
    q = torch.randn((tokens, heads, dim), generator=g, device=DEV).bfloat16()
    table = torch.arange(tokens * blocks, dtype=torch.int32, device=DEV).view(tokens, blocks)
    at = torch.full((tokens,), keys - 1, dtype=torch.int32, device=DEV)
    seq = torch.arange(tokens, dtype=torch.int32, device=DEV)
    return lambda: ops.cached_attention(q, *cache, at, seq, table, heads, dim, dim, dim ** -0.5,
                                        heads_first=True, key_splits=4)


@pytest.mark.gpu
@pytest.mark.parametrize("dim", [80, 96, 256])
def test_two_attentions_side_by_side(dim):
    """Two calls whose blocks count how many of them are done, one in a branch: the same bits as one after
    the other, whatever the count that calls in plain order share holds meanwhile."""
    left, right = attention_case(dim, 1), attention_case(dim, 2)
    want = [left().clone(), right().clone()]

    def both():
        with ops.aside(right, STEP, 2) as beside:
            first = left()
        return first, beside.result

    graph, out = captured(both)
    shared = ops._attention_tickets[out[0].device]
    shared.fill_(12345)          # (blocks that counted here would never be the last ones)
    try:
        for _ in range(20):
            graph.replay()
            assert torch.equal(out[0], want[0]) and torch.equal(out[1], want[1])
            out[0].zero_(), out[1].zero_()
    finally:
        shared.zero_()
    assert torch.equal(left(), want[0])


@pytest.mark.gpu
def test_the_library_s_workspace_is_not_shared_by_branches(monkeypatch):
    """Products that only the library takes (rows of no whole 16 bytes), added into a stream."""
    g = torch.Generator(device=DEV).manual_seed(3)
    x, w = (torch.randn(s, 12, generator=g, device=DEV).bfloat16() for s in (4, 20))
    spaces = []
    monkeypatch.setattr(sys.modules[ops.linear.__module__], "call", lambda name, *args: (
        spaces.append(args[8]) if name == "sakv_lib_accumulate" else None, _lib.call(name, *args)))

    def product():
        return ops.linear(x, w, accumulate_into=torch.ones((4, 20), device=DEV))

    def both():
        spaces.clear()
        with ops.aside(product, STEP, 4) as beside:
            first = product()
        return first, beside.result, product()

    graph, out = captured(both)
    assert len(set(spaces)) == len(spaces) == 3
    graph.replay()
    want = 1 + x.double() @ w.double().T
    for y in out:                                            # (12 products, fp32)
        assert ((y.double() - want).abs() <= 16 * 2.0 ** -23 * (1 + want.abs())).all()


def small(x):
    """Some of this library's kernels with temporaries that come and go."""
    y = ops.linear(x, x, out_dtype=torch.float32)
    ops.add_into(y, ops.linear(x, x, out_dtype=torch.float32))
    return ops.linear(y.bfloat16(), x.T.contiguous(), out_dtype=torch.float32)


@pytest.mark.gpu
def test_a_branch_inside_a_branch():
    """An outer and an inner branch in turn, twice, what they made given back in between: the bits of the
    same calls one after the other."""
    g = torch.Generator(device=DEV).manual_seed(5)
    xs = [torch.randn(64, 64, generator=g, device=DEV).bfloat16() for _ in range(6)]

    def outer(a, b):
        with ops.aside(lambda: small(a), STEP, 64) as inner:
            own = small(b)
        return own + inner.result

    def step():
        outs = []
        for a, b, c in (xs[:3], xs[3:]):
            with ops.aside(lambda: outer(a, b), STEP, 64) as beside:
                own = small(c)
            outs.append(own - beside.result)
            del own, beside
        return outs

    want = [y.clone() for y in step()]
    graph, out = captured(step)
    for _ in range(10):
        graph.replay()
        for y, w in zip(out, want):
            assert torch.equal(y, w)
            y.zero_()


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["in the branch", "beside it", "in an inner branch"])
def test_a_failure_ends_the_branch(where):
    """What fails inside a capture is what the caller sees; afterwards everything works as before."""
    x = torch.ones(64, 64, device=DEV).bfloat16()

    def failing():
        ops.linear(x, x)
        raise ops.KernelError("a part says no")

    def inner():
        with ops.aside(failing, STEP, 64):
            return small(x)

    def step():
        first = {"in the branch": failing, "beside it": lambda: small(x), "in an inner branch": inner}[where]
        with ops.aside(first, STEP, 64):
            return failing() if where == "beside it" else small(x)

    small(x)
    torch.cuda.synchronize()
    with pytest.raises(ops.KernelError, match="a part says no"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            step()
    assert not apart()

    def fine():
        with ops.aside(lambda: small(x), STEP, 64) as beside:
            own = small(x)
        return own, beside.result

    graph, out = captured(fine)
    graph.replay()
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], small(x))


@pytest.mark.gpu
def test_a_branch_s_stream_is_its_thread_s_own():
    """No two threads', and none that PyTorch deals out; a thread that has ended leaves its streams to the next."""
    from concurrent.futures import ThreadPoolExecutor
    main = torch.cuda.current_stream()

    def mine():
        first = branch._other_stream(main)
        return first.cuda_stream, branch._other_stream(first).cuda_stream

    dealt = {torch.cuda.Stream().cuda_stream for _ in range(80)}
    meet = threading.Barrier(3, timeout=60)

    def held():
        both = mine()
        meet.wait()
        assert mine() == both
        return both

    with ThreadPoolExecutor(3) as pool:
        taken = [s for f in [pool.submit(held) for _ in range(3)] for s in f.result()]
    assert len(set(taken)) == 6 and not dealt & set(taken)
    gc.collect()
    with ThreadPoolExecutor(1) as pool:
        again = pool.submit(mine).result()
    assert set(again) <= set(taken)
