"""A prompt in runs (csrc/chunk_scan.cu and the selective scan's run kernels) at the edges of a run and of
its tiles, and with values that are not finite: nothing before such a value's token may feel it."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

from semantic_aware_adaptive_kv_cache_precision_b200 import ops

pytestmark = pytest.mark.gpu

DEV = "cuda"


def step_of(lengths):
    at = torch.tensor([0, *lengths]).cumsum(0).int().to(DEV)
    return SimpleNamespace(sequences=len(lengths), max_new=max(lengths), cu_seqlens=at, is_decode=False,
                           slots=torch.arange(len(lengths), dtype=torch.int32, device=DEV),
                           positions=torch.cat([torch.arange(n) for n in lengths]).int().to(DEV))


def walked(decay, d, k, v, q, lengths):
    """[T, heads, vdim] and the last states, in 64 bits: decay, d [T, heads]; k, q [T, heads, dim]."""
    outs, states, at = [], [], 0
    for n in lengths:
        S = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=torch.float64, device=DEV)
        for t in range(at, at + n):
            S = decay[t][:, None, None] * S + (d[t][:, None] * k[t])[:, :, None] * v[t][:, None]
            outs.append(torch.einsum("hkv,hk->hv", S, q[t]))
        at += n
        states.append(S.transpose(1, 2))
    return torch.stack(outs), torch.stack(states)


def fading(proj, heads, dim, vdim, less_one, lengths, run):
    state = torch.zeros(len(lengths), heads, vdim, dim, device=DEV)
    out = ops.decay_attention(proj, 0, heads * dim, 2 * heads * dim, heads, dim, vdim, less_one, state,
                              step_of(lengths), run=run, activation=False)
    return out.view(-1, heads, vdim), state


# fp32 sums of a few hundred products in another order than 64 bits adds them: some units of 2^-24 of
# the largest of them; ten such units as everywhere in these tests' neighbours (2e-5) are far more
TOL = 2e-5


@pytest.mark.parametrize("lengths,run", [((1, 64, 65), 64), ((63, 127, 128), 64), ((129, 2), 64),
                                         ((16, 17, 33), 16), ((50, 7), 13), ((200,), 100)])
@pytest.mark.parametrize("dim,vdim", [(16, 16), (17, 3), (64, 65), (128, 64), (100, 130), (256, 8)])
def test_a_run_s_edges(lengths, run, dim, vdim):
    heads, T = 2, sum(lengths)
    g = torch.Generator(device=DEV).manual_seed(T + dim + vdim)
    proj = torch.randn(T, heads * (2 * dim + vdim), generator=g, device=DEV)
    less_one = torch.tensor([-0.0625, -0.5], device=DEV)
    got, state = fading(proj, heads, dim, vdim, less_one, lengths, run)
    p = proj.double()
    q, k = (p[:, i * heads * dim:(i + 1) * heads * dim].view(T, heads, dim) for i in (0, 1))
    decay = (1 + less_one.double()).expand(T, heads)
    want, last = walked(decay, torch.ones_like(decay), k, p[:, 2 * heads * dim:].view(T, heads, vdim), q,
                        lengths)
    for a, b in ((got, want), (state, last)):
        assert (a.double() - b).abs().max() <= TOL * b.abs().max()


@pytest.mark.parametrize("lengths,run", [((64, 131, 1), 64), ((100, 33), 32)])
def test_decays_of_any_sign_and_size(lengths, run):
    """Decays below zero change the state's sign with every token; a decay of zero forgets it at once."""
    heads, dim, vdim, T = 6, 24, 20, sum(lengths)
    g = torch.Generator(device=DEV).manual_seed(T)
    proj = torch.randn(T, heads * (2 * dim + vdim), generator=g, device=DEV)
    less_one = torch.tensor([-1.5, -1.96875, -1.0, -2.0, 0.0, 0.015625], device=DEV)     # -0.5, -0.97, 0, -1, 1 ...
    got, state = fading(proj, heads, dim, vdim, less_one, lengths, run)
    p = proj.double()
    q, k = (p[:, i * heads * dim:(i + 1) * heads * dim].view(T, heads, dim) for i in (0, 1))
    v = p[:, 2 * heads * dim:].view(T, heads, vdim)
    decay = (1 + less_one.double()).expand(T, heads)
    one = torch.ones_like(decay)
    want, last = walked(decay, one, k, v, q, lengths)
    bound, last_bound = walked(decay.abs(), one, k.abs(), v.abs(), q.abs(), lengths)
    assert ((got.double() - want).abs() <= TOL * bound).all()
    assert ((state.double() - last).abs() <= TOL * last_bound).all()


@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3.4e38])
@pytest.mark.parametrize("where", ["key", "value", "query"])
def test_a_value_that_is_not_finite_is_not_felt_before(value, where):
    heads, dim, vdim, n, at = 2, 64, 96, 150, 75
    g = torch.Generator(device=DEV).manual_seed(7)
    proj = torch.randn(n, heads * (2 * dim + vdim), generator=g, device=DEV)
    less_one = torch.tensor([-0.01, -0.3], device=DEV)
    clean, _ = fading(proj, heads, dim, vdim, less_one, (n,), 64)
    column = {"query": 5, "key": heads * dim + 5, "value": 2 * heads * dim + 5}[where]    # of head 0
    proj[at, column] = value
    got, _ = fading(proj, heads, dim, vdim, less_one, (n,), 64)
    one, _ = fading(proj, heads, dim, vdim, less_one, (n,), 0)           # token by token
    assert torch.equal(got[:64], clean[:64]) and torch.equal(got[:, 1], clean[:, 1])
    assert (got[:at] - clean[:at]).abs().max() <= TOL * clean.abs().max()
    same = torch.isfinite(got) == torch.isfinite(one)
    assert same.all()
    ok = torch.isfinite(one)
    assert (got[ok] - one[ok]).abs().max() <= TOL * one[ok].abs().max()


@pytest.mark.parametrize("lengths,run", [((1, 64, 65), 64), ((200, 31), 64), ((40, 17), 16)])
@pytest.mark.parametrize("channels,n_state,rank", [(128, 16, 16), (130, 16, 40), (37, 9, 7), (300, 15, 256)])
def test_selective_scan_in_runs(lengths, run, channels, n_state, rank):
    T = sum(lengths)
    g = torch.Generator(device=DEV).manual_seed(T + channels)
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)
    x, low, z = rand(T, channels).bfloat16(), 0.3 * rand(T, rank + 2 * n_state), rand(T, channels)
    w, b = (0.1 * rand(channels, rank)).bfloat16(), (rand(channels) - 2).bfloat16()
    a_log, skip = rand(channels, n_state).bfloat16(), rand(channels).bfloat16()
    dt = ops.step_size(low, rank, w, b)
    exact = torch.nn.functional.softplus(low[:, :rank].double() @ w.double().T + b.double())
    assert (dt.double() - exact).abs().max() <= TOL * exact.abs().max()
    state = torch.zeros(len(lengths), channels, n_state, device=DEV)
    got = ops.selective_scan(x, dt, low, rank, rank + n_state, n_state, z, a_log, skip, state,
                             step_of(lengths), run=run)
    A, d, at, outs, states = -torch.exp(a_log.double()), dt.double(), 0, [], []
    B, C = low[:, rank:rank + n_state].double(), low[:, rank + n_state:].double()
    for n in lengths:
        S = torch.zeros(channels, n_state, dtype=torch.float64, device=DEV)
        for t in range(at, at + n):
            S = torch.exp(d[t][:, None] * A) * S + (d[t] * x[t].double())[:, None] * B[t]
            outs.append((S @ C[t] + skip.double() * x[t].double()) * torch.nn.functional.silu(z[t].double()))
        at += n
        states.append(S)
    want, last = torch.stack(outs), torch.stack(states)
    assert (state.double() - last).abs().max() <= TOL * last.abs().max()
    assert (got.double() - want).abs().max() <= 2.0 ** -8 * want.abs().max()     # (rounded once to 16 bits)


@pytest.mark.parametrize("lengths,run", [((300, 90), 64), ((100,), 32)])
def test_what_a_run_forgets_leaves_no_rest(lengths, run):
    """One very large token early in a sequence, strong decays and small tokens after it: every number's
    error is bounded by the sum of what it is made of (the same recurrence over absolute values), not by
    the largest number of the step. (Such a bound is what fp32 sums in any order keep; a state taken off
    itself keeps an ulp of what it was.)"""
    heads, dim, vdim, T = 2, 32, 40, sum(lengths)
    g = torch.Generator(device=DEV).manual_seed(T)
    proj = 0.1 * torch.randn(T, heads * (2 * dim + vdim), generator=g, device=DEV)
    at = 0
    for n in lengths:
        proj[at + 3] *= 1e4
        at += n
    less_one = torch.tensor([-0.25, -0.375], device=DEV)
    got, state = fading(proj, heads, dim, vdim, less_one, lengths, run)
    p = proj.double()
    q, k = (p[:, i * heads * dim:(i + 1) * heads * dim].view(T, heads, dim) for i in (0, 1))
    v = p[:, 2 * heads * dim:].view(T, heads, vdim)
    decay = (1 + less_one.double()).expand(T, heads)
    one = torch.ones_like(decay)
    want, last = walked(decay, one, k, v, q, lengths)
    bound, last_bound = walked(decay, one, k.abs(), v.abs(), q.abs(), lengths)
    assert ((got.double() - want).abs() <= TOL * bound).all()
    assert ((state.double() - last).abs() <= TOL * last_bound).all()

    # the dual form and the selective scan, whose tokens choose how much is forgotten
    dt = torch.full((T, heads), 0.5, device=DEV)
    a, zero = torch.tensor([-0.6, -1.3], device=DEV), torch.zeros(heads, device=DEV)
    xbc = torch.cat([v[:, :].reshape(T, -1).float(), k[:, 0].float(), q[:, 0].float()], 1).contiguous()
    state = torch.zeros(len(lengths), heads, vdim, dim, device=DEV)
    got = ops.dual_scan(xbc, 0, heads * vdim, heads * vdim + dim, dt, zero, a, zero, heads, 1, dim, vdim,
                        state, step_of(lengths), run=run).view(T, heads, vdim)
    d = torch.nn.functional.softplus(dt.double())
    decay = torch.exp(d * a.double())
    k1, q1 = (z[:, :1].expand(T, heads, dim) for z in (k, q))
    want, last = walked(decay, d, k1, v, q1, lengths)
    bound, last_bound = walked(decay, d, k1.abs(), v.abs(), q1.abs(), lengths)
    assert ((got.double() - want).abs() <= TOL * bound).all()
    assert ((state.double() - last).abs() <= TOL * last_bound).all()

    channels, n_state = 64, 16
    x = torch.ones(T, channels, device=DEV)
    at = 0
    for n in lengths:
        x[at + 3] = 1e4
        at += n
    x = x.bfloat16()
    low = 0.1 * torch.rand(T, 2 * n_state, generator=g, device=DEV)
    dt = torch.full((T, channels), 0.75, device=DEV)
    a_log = torch.zeros(channels, n_state, device=DEV)
    state = torch.zeros(len(lengths), channels, n_state, device=DEV)
    ops.selective_scan(x, dt, low, 0, n_state, n_state, torch.ones(T, channels, device=DEV), a_log,
                       torch.zeros(channels, device=DEV), state, step_of(lengths), run=run)
    fade = torch.exp(-dt[0, 0].double())                     # (all terms are positive)
    at = 0
    for b, n in enumerate(lengths):
        S = torch.zeros(channels, n_state, dtype=torch.float64, device=DEV)
        for t in range(at, at + n):
            S = fade * S + dt[t].double()[:, None] * x[t].double()[:, None] * low[t, :n_state].double()
        at += n
        assert ((state[b].double() - S).abs() <= TOL * S).all()


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38])
@pytest.mark.parametrize("where", ["low", "weight"])
def test_step_sizes_of_values_that_are_not_finite(value, where):
    """On the tensor cores as number by number (the kernel for fp32 weights): the same numbers are not
    finite, and in the same way."""
    T, channels, rank = 70, 66, 40
    g = torch.Generator(device=DEV).manual_seed(11)
    low = torch.randn(T, rank + 4, generator=g, device=DEV)
    w = (0.3 * torch.randn(channels, rank, generator=g, device=DEV)).bfloat16()
    b = torch.randn(channels, generator=g, device=DEV).bfloat16()
    w[5, 3] = 0.0
    if where == "low":
        low[17, 3], low[69, 39] = value, value
    else:
        w[9, 3], w[65, 39] = value, value             # (3.4e38 is infinite in 16 bits)
    got = ops.step_size(low, rank, w, b)
    want = ops.step_size(low, rank, w.float(), b.float())
    odd = ~torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), ~odd)
    assert torch.equal(got[odd].nan_to_num(nan=-1.0), want[odd].nan_to_num(nan=-1.0))
    assert ((got[~odd] - want[~odd]).abs() <= TOL * (8 + want[~odd].abs())).all()      # (sums of some units)
