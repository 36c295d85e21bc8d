"""Cached attention on the tensor cores (`csrc/attention_mma.cu`): the rule that sends calls to it
(no GPU needed), and its results against float64 and against the general kernel at the edges of its
tiles, in prompts, pieces, steps of scattered tokens and decoded, with infinities among the values."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from semantic_aware_adaptive_kv_cache_precision_b200 import ops
from semantic_aware_adaptive_kv_cache_precision_b200.ops import attention_mma
from semantic_aware_adaptive_kv_cache_precision_b200.parts.distance_attention import LogDistanceAttention

BF = torch.bfloat16


def test_only_bfloat16_rows_at_multiples_of_16_bytes_go_to_the_tensor_cores():
    def asks(dtype=BF, dim=128, vdim=128, maps=1, stride=2048, offset=0, head=None, k_row=None,
             latent=False, q2=None, split=0):
        q = torch.zeros(8 * stride + 8, dtype=dtype)[offset:][:4 * stride].view(4, stride)
        k = torch.zeros((1, 1, 64, k_row or maps * dim), dtype=dtype)
        v = None if latent else torch.zeros((1, 1, 64, vdim), dtype=dtype)
        return attention_mma.takes(q, head or dim, k, v, dim, vdim, maps, q2, split)

    assert asks() and asks(dim=64, vdim=64) and asks(vdim=256, maps=2) and asks(maps=2)
    assert asks(dim=576, vdim=512, latent=True) and asks(offset=8) and asks(stride=2056)
    q2 = torch.zeros((4, 4, 64), dtype=BF)
    assert asks(dim=576, vdim=512, latent=True, q2=q2, split=512)
    assert not asks(dim=576, vdim=512, latent=True, q2=q2, split=511)
    wide = torch.zeros(4 * 4 * 69, dtype=BF).view(4, 4, 69)
    assert not asks(dim=576, vdim=512, latent=True, q2=wide[:, :, 5:], split=512)
    assert not asks(dtype=torch.float32) and not asks(dim=96) and not asks(vdim=64)
    assert not asks(dim=64, vdim=64, maps=2) and not asks(offset=3) and not asks(stride=2052)
    assert not asks(head=132) and not asks(k_row=132) and not asks(dim=128, vdim=128, latent=True)


def test_attention_beside_library_products_is_launched_in_plain_order(monkeypatch):
    """Only the attention with the logarithmic penalty, whose neighbours are this library's own
    kernels, may be overlapped with them."""
    launched = []
    monkeypatch.setattr(attention_mma, "call", lambda name, *args: launched.append((name, args[-1])))
    monkeypatch.setattr(ops, "require_cuda", lambda *tensors: None)
    pos, table = torch.zeros(3, dtype=torch.int32), torch.zeros((1, 1), dtype=torch.int32)

    def cache(width):
        return torch.zeros((1, 1, 64, width), dtype=BF)

    for form in ({}, {"heads_first": True, "key_splits": 2}):
        ops.cached_attention(torch.zeros((3, 4, 576), dtype=BF), cache(576), None, pos, pos, table, 4, 576, 512,
                             1.0, **form)
        ops.cached_attention(torch.zeros((3, 4, 128), dtype=BF), cache(256), cache(256), pos, pos, table, 2, 128,
                             256, 1.0, maps=2, **form)
        ops.cached_attention(torch.zeros((3, 4, 128), dtype=BF), cache(128), cache(128), pos, pos, table, 4, 128,
                             128, 1.0, **form)
    assert launched == [("sakv_attention_mma", 1)] * 6
    slope = torch.zeros(4)
    ops.distance_attention(torch.zeros((3, 1024), dtype=BF), cache(128), cache(128), pos, pos, table, 4, 1.0, None,
                           slope, slope)
    assert launched[6:] == [("sakv_attention_mma", 0)]


def test_only_calls_that_the_tensor_cores_take_have_their_splits_bounded_by_blocks(monkeypatch):
    """Gates of an odd number of heads behind the queries, keys and values leave rows that do not begin at
    multiples of 16 bytes: those go to the general kernel, whose splits are warps."""
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    spec = SimpleNamespace(head_dim=128, value_dim=128, window=None, heads=6, kv_heads=2)
    step = SimpleNamespace(is_decode=True, max_len_bound=4096, max_len=4096, tokens=64)
    cache = torch.zeros((1, 2, 64, 128), dtype=BF)
    view = SimpleNamespace(keys=cache, values=cache)

    def splits(columns, dtype=BF):
        return LogDistanceAttention._splits(SimpleNamespace(spec=spec), step,
                                            torch.zeros((64, columns), dtype=dtype), view)

    assert splits(10 * 128) == 4 and splits(10 * 128 + 6) == 16 and splits(10 * 128, torch.float32) == 1
    step.tokens = 1
    assert splits(10 * 128) == 16
    spec.head_dim = 96
    step.tokens = 64
    assert splits(1280) == 16


def case(seed, lens, heads, kv_heads, dim, vdim, maps=1, latent=False):
    """Sequences of `lens` tokens in a cache whose unused positions hold NaN."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def draw(*shape):
        return torch.randn(shape, generator=g, device="cuda").to(BF)

    blocks = [-(-n // 64) for n in lens]
    total, k_row = sum(blocks) + 1, maps * dim
    keys = torch.full((total, kv_heads, 64, k_row), float("nan"), dtype=BF, device="cuda")
    values = None if latent else torch.full((total, kv_heads, 64, vdim), float("nan"), dtype=BF,
                                            device="cuda")
    table = torch.zeros((len(lens), max(blocks)), dtype=torch.int32)
    order, at, rows = np.random.default_rng(seed).permutation(total), 0, []
    for i, n in enumerate(lens):
        table[i, :blocks[i]] = torch.as_tensor(order[at:at + blocks[i]])
        at += blocks[i]
        k, v = draw(n, kv_heads, k_row), draw(n, kv_heads, vdim)
        for p in range(0, n, 64):
            b, m = int(table[i, p // 64]), min(64, n - p)
            keys[b, :, :m] = k[p:p + m].transpose(0, 1)
            if not latent:
                values[b, :, :m] = v[p:p + m].transpose(0, 1)
        rows.append((k, k[:, :, :vdim] if latent else v))
    return draw, keys, values, table.cuda(), rows


def in_64_bits(q, pos, seq, rows, heads, kv_heads, dim, maps, scale, window=0, chunk=0, keep=0,
               sink=None, softcap=None, linear=None, slope=None, rate=None, lam=0.0, eps=0.0):
    out = []
    for t, (p, s) in enumerate(zip(pos, seq)):
        k, v = rows[s][0][:p + 1].double(), rows[s][1][:p + 1].double()
        j = torch.arange(p + 1, device="cuda")
        seen = torch.ones_like(j, dtype=torch.bool)
        if window:
            seen = (p - j < window) | (j < keep)
        if chunk:
            seen = j // chunk == p // chunk
        dist = (p - j).double()
        for h in range(heads):
            g, a = h // (heads // kv_heads), []
            for m in range(maps):
                x = k[:, g, m * dim:(m + 1) * dim] @ q[t, h * maps + m].double() * scale
                if softcap:
                    x = softcap * torch.tanh(x / softcap)
                if slope is not None:
                    x = x - slope[h].double() * torch.log1p(rate[h].double() * dist)
                if linear is not None:
                    x = x - linear[h].double() * dist
                x = x.masked_fill(~seen, -float("inf"))
                if sink is not None:
                    x = torch.cat([x, sink[h].double().reshape(1)])
                a.append(torch.softmax(x, 0)[:p + 1][seen] @ v[seen, g])
            y = a[0]
            if maps == 2:
                y = a[0] - lam * a[1]
                y = y / torch.sqrt((y * y).mean() + eps)
            out.append(y)
    return torch.stack(out).view(len(pos), -1)


def near(got, want, rel=2.0 ** -8):
    """Rounding to bfloat16 alone leaves up to 2^-8 of a value; sums in fp32 and weights of 16 bits
    add under a hundredth of that. Against another kernel's bfloat16 numbers: a step of the type,
    which is up to 2^-7 of a value."""
    worst = float(((got.double() - want).abs() - rel * want.abs()).max())
    assert worst <= 1e-4 * float(want.abs().max()), worst


STEPS = {                                # (position, sequence) of every token of a step
    "prompt": [(p, 0) for p in range(97)],
    "two prompts": [(p, 0) for p in range(70)] + [(p, 1) for p in range(33)],
    "a piece": [(p, 0) for p in range(61, 131)],
    "one token": [(130, 0)],
    "scattered": [(5, 1), (6, 1), (128, 0), (129, 0), (3, 0), (64, 0), (63, 0), (0, 1)],
}


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,maps,latent,more", [
    (6, 2, 64, 64, 1, False, {}), (8, 2, 128, 128, 1, False, {"window": 50, "keep": 3, "sink": True}),
    (5, 1, 128, 128, 1, False, {"softcap": 9.0, "linear": True}), (4, 4, 128, 128, 1, False, {"slope": True}),
    (20, 1, 64, 64, 1, False, {"window": 64}), (4, 2, 128, 256, 2, False, {"chunk": 48}),
    (3, 1, 128, 128, 2, False, {}), (40, 1, 128, 128, 2, False, {"window": 50, "keep": 3, "sink": True}),
    (35, 1, 128, 256, 2, False, {"softcap": 9.0, "linear": True}), (2, 1, 128, 256, 1, False, {"window": 1}),
    (16, 1, 576, 512, 1, True, {"window": 70, "sink": True}), (3, 1, 576, 512, 1, True, {"chunk": 65})])
def test_the_edges_of_tiles_in_every_kind_of_step(heads, kv_heads, dim, vdim, maps, latent, more):
    draw, keys, values, table, rows = case(heads + dim, (131, 40), heads, kv_heads, dim, vdim, maps, latent)
    more = dict(more)
    u = torch.rand(heads, device="cuda")
    sink = 2 * u if more.pop("sink", False) else None
    linear = 0.1 * u if more.pop("linear", False) else None
    slope, rate = (2 * u, 0.1 + 0.4 * u) if more.pop("slope", False) else (None, None)
    scale = 1.5 * dim ** -0.5
    for name, step in STEPS.items():
        pos, seq = [p for p, _ in step], [s for _, s in step]
        q = draw(len(step), heads * maps, dim)
        want = in_64_bits(q, pos, seq, rows, heads, kv_heads, dim, maps, scale, sink=sink, linear=linear,
                          slope=slope, rate=rate, lam=0.4, eps=1e-6, **more)
        positions = torch.tensor(pos, dtype=torch.int32, device="cuda")
        token_seq = torch.tensor(seq, dtype=torch.int32, device="cuda")
        for splits in (0, 1, 2, 5):                      # 0: a prompt's form
            got = attention_mma.attention(
                q, dim, keys, values, positions, token_seq, table, heads, dim, vdim, scale, maps=maps,
                window=more.get("window"), chunk=more.get("chunk"), keep_first=more.get("keep", 0),
                slope=slope, rate=rate, softcap=more.get("softcap"), linear=linear, sink=sink, lam=0.4,
                eps=1e-6, decode=splits > 0, key_splits=max(1, splits))
            near(got, want)
        alone = attention_mma.attention(
            q[-1:], dim, keys, values, positions[-1:], token_seq[-1:], table, heads, dim, vdim, scale,
            maps=maps, window=more.get("window"), chunk=more.get("chunk"),
            keep_first=more.get("keep", 0), slope=slope, rate=rate, softcap=more.get("softcap"),
            linear=linear, sink=sink, lam=0.4, eps=1e-6)
        counts = [seq.count(0), seq.count(1)]
        cu = torch.tensor([0, counts[0], len(seq)], dtype=torch.int32, device="cuda")
        together = {}
        for told in (False, True):              # (tokens that lie sequence by sequence: told, or found out)
            if told and seq != [0] * counts[0] + [1] * counts[1]:
                continue
            together[told] = attention_mma.attention(
                q, dim, keys, values, positions, token_seq, table, heads, dim, vdim, scale, maps=maps,
                window=more.get("window"), chunk=more.get("chunk"), keep_first=more.get("keep", 0),
                slope=slope, rate=rate, softcap=more.get("softcap"), linear=linear, sink=sink, lam=0.4,
                eps=1e-6, cu_seqlens=cu if told else None)
            assert torch.equal(alone[0], together[told][-1]), name      # whatever came with it: the same bits
        if True in together:
            assert torch.equal(together[True], together[False]), name


@pytest.mark.gpu
@pytest.mark.parametrize("dim,vdim,maps,latent", [(128, 128, 1, False), (128, 256, 2, False), (576, 512, 1, True)])
@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan")])
def test_a_value_that_is_not_finite_reaches_the_rows_that_see_it_and_no_others(dim, vdim, maps, latent, value,
                                                                               monkeypatch):
    """Position 70 of 131 holds it in one column: rows before it are as without it, rows from it on
    are what the general kernel gives, and other columns are as without it (over a latent row the
    key is the value, so the rows from it on have no number at all)."""
    heads = 4
    draw, keys, values, table, _ = case(3, (131,), heads, 1, dim, vdim, maps, latent)
    q = draw(131, heads * maps, dim)
    pos = torch.arange(131, dtype=torch.int32, device="cuda")
    seq = torch.zeros(131, dtype=torch.int32, device="cuda")

    def run(lo=0, **form):
        return ops.cached_attention(q[lo:], keys, values, pos[lo:], seq[lo:], table, heads, dim, vdim,
                                    dim ** -0.5, maps=maps, lam=0.4, eps=1e-6, **form)

    forms = (dict(), dict(lo=128, heads_first=True, key_splits=1), dict(lo=128, heads_first=True, key_splits=3))
    clean = [run(**f) for f in forms]
    (keys if latent else values)[table[0, 1].long(), 0, 6, 9] = value
    for before, form in zip(clean, forms):
        got = run(**form)
        with monkeypatch.context() as m:
            m.setattr(attention_mma, "takes", lambda *a, **k: False)
            general = run(**form)
        lo = form.get("lo", 0)
        early = max(0, 70 - lo)
        if early:
            near(got[:early], before[:early].double(), 2.0 ** -7)
            assert bool(torch.isfinite(got[:early]).all())
        assert torch.equal(torch.isnan(got), torch.isnan(general))
        assert torch.equal(torch.isinf(got), torch.isinf(general))
        same = torch.isfinite(general)
        if bool(same.any()):
            near(got[same], general[same].double(), 2.0 ** -7)


@pytest.mark.gpu
@pytest.mark.parametrize("penalty", ["none", "linear", "logarithm"])
@pytest.mark.parametrize("splits", [0, 1, 2])
def test_weights_and_penalties_keep_their_32_bits(penalty, splits):
    """Two keys whose values nearly cancel: (p0 - c p1) / (p0 + p1), c a bfloat16 number near p0 / p1.
    What is left shows an error of the weights that rounding the output (2^-8 of it) does not hide: with
    fp32 weights some 2^-23, with weights of 16 bits or a penalty as log2(1 + x) up to 2^-19 and more."""
    heads, dim = 64, 128
    g = torch.Generator(device="cuda").manual_seed(splits)
    q = torch.zeros((1, heads, dim), dtype=BF, device="cuda")
    keys = torch.zeros((1, 1, 64, dim), dtype=BF, device="cuda")
    values = torch.zeros_like(keys)
    gap = 0.01 + 0.05 * torch.rand(heads, generator=g, device="cuda")        # of the two scores
    linear = slope = rate = None
    distance = torch.tensor([1.0, 0.0], dtype=torch.float64, device="cuda")
    if penalty == "none":
        keys[0, 0, 0, 0] = 1.0
        q[0, :, 0] = -gap.to(BF)
        scores = torch.outer(q[0, :, 0].double(), distance)
    elif penalty == "linear":
        linear = gap
        scores = -torch.outer(gap.double(), distance)
    else:
        rate = torch.full((heads,), 1.37 * 2.0 ** -13, device="cuda")
        slope = gap / rate
        scores = -slope.double()[:, None] * torch.log1p(torch.outer(rate.double(), distance))
    c = (1 + torch.arange(dim, device="cuda") / dim / 14).to(BF)
    values[0, 0, 0], values[0, 0, 1] = c, -1.0
    want = torch.softmax(scores, 1) @ torch.stack([c.double(), -torch.ones_like(c).double()])
    zero = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = attention_mma.attention(q, dim, keys, values, zero + 1, zero, zero[:, None], heads, dim, dim, 1.0,
                                  slope=slope, rate=rate, linear=linear, decode=splits > 0,
                                  key_splits=max(1, splits))
    off = (got.view(heads, dim).double() - want).abs() - 2.0 ** -8 * want.abs()
    assert float(off.max()) <= 2.0 ** -21


@pytest.mark.gpu
@pytest.mark.parametrize("first,window", [(0, None), (64, None), (91, 40), (100, 31)])
def test_a_first_key_that_scores_minus_infinity_counts_for_nothing(first, window):
    """The key at `first` (a sequence's, a split's or some windows' first) scores -inf with every query; an
    infinite value at position 110 sends the blocks that see it through their keys one by one."""
    heads, dim, n = 4, 128, 131
    draw, keys, values, table, rows = case(5, (n,), heads, 1, dim, dim)
    q = draw(n, heads, dim)
    q[:, :, 9] = -q[:, :, 9].abs() - 0.1
    keys[table[0, first // 64].long(), 0, first % 64, 9] = float("inf")
    values[table[0, 1].long(), 0, 110 - 64, 3] = float("inf")
    k, v = rows[0][0].clone(), rows[0][1].clone()
    k[first, 0, 9], v[110, 0, 3] = float("inf"), float("inf")
    pos = torch.arange(n, dtype=torch.int32, device="cuda")
    seq = torch.zeros_like(pos)
    want = in_64_bits(q, range(n), [0] * n, [(k, v)], heads, 1, dim, 1, dim ** -0.5, window=window or 0)
    for lo, splits in ((0, 0), (128, 1), (128, 3), (130, 2)):
        got = attention_mma.attention(q[lo:], dim, keys, values, pos[lo:], seq[lo:], table, heads, dim, dim,
                                      dim ** -0.5, window=window, decode=splits > 0,
                                      key_splits=max(1, splits))
        same = torch.isfinite(want[lo:])
        assert torch.equal(torch.isnan(got), torch.isnan(want[lo:]))
        assert torch.equal(torch.isinf(got), torch.isinf(want[lo:]))
        near(got[same], want[lo:][same])


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,maps,latent", [(8, 2, 128, 128, 1, False), (4, 4, 64, 64, 1, False),
                                                                 (4, 2, 128, 256, 2, False), (16, 1, 576, 512, 1, True)])
def test_tokens_of_several_sequences_in_one_step_run_side_by_side(heads, kv_heads, dim, vdim, maps, latent):
    """Fifteen tokens that each continue a sequence of its own beside a piece of a prompt, as a scheduler
    mixes them: the rows fit a few tiles, and walked one after another in those tiles' blocks they took
    many times what one of them takes alone."""
    lens = [3000 + 7 * i for i in range(15)] + [200]
    draw, keys, values, table, _ = case(8, lens, heads, kv_heads, dim, vdim, maps, latent)
    pos = [n - 1 for n in lens[:15]] + list(range(100, 200))
    seq = list(range(15)) + [15] * 100
    q = draw(len(pos), heads * maps, dim)
    positions = torch.tensor(pos, dtype=torch.int32, device="cuda")
    token_seq = torch.tensor(seq, dtype=torch.int32, device="cuda")
    cu = torch.tensor(list(range(16)) + [115], dtype=torch.int32, device="cuda")

    def run(n, cu_seqlens):
        return attention_mma.attention(q[:n], dim, keys, values, positions[:n], token_seq[:n], table, heads, dim,
                                       vdim, dim ** -0.5, maps=maps, lam=0.3, eps=1e-6, cu_seqlens=cu_seqlens)

    def time(n, cu_seqlens):
        best = float("inf")
        for _ in range(5):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            run(n, cu_seqlens)
            begin.record()
            for _ in range(10):
                run(n, cu_seqlens)
            end.record()
            end.synchronize()
            best = min(best, begin.elapsed_time(end))
        return best

    alone = time(1, cu.clamp(max=1))
    assert time(115, cu) < 3 * alone and time(115, None) < 3 * alone
    assert torch.equal(run(115, cu), run(115, None)) and torch.equal(run(1, cu.clamp(max=1)), run(115, cu)[:1])


@pytest.mark.gpu
@pytest.mark.parametrize("vdim", [128, 256])
def test_a_prompt_of_two_maps_needs_no_memory_beside_its_output(vdim):
    heads, dim, n = 8, 128, 2000
    draw, keys, values, table, _ = case(4, (n,), heads, 2, dim, vdim, 2)
    q = draw(n, 2 * heads, dim)
    pos = torch.arange(n, dtype=torch.int32, device="cuda")
    zeros = torch.zeros_like(pos)

    def run():
        return ops.cached_attention(q, keys, values, pos, zeros, table, heads, dim, vdim, dim ** -0.5, maps=2,
                                    lam=0.4, eps=1e-6)

    run()
    torch.cuda.synchronize()
    held = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    out = run()
    torch.cuda.synchronize()
    assert torch.cuda.max_memory_allocated() - held <= out.numel() * 2 + 4096
