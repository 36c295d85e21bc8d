"""Kernels that choose a form by the sizes of a call: every form against float64, and against one
another where the result must not depend on the form."""

from types import SimpleNamespace

import pytest
import torch

from semantic_aware_adaptive_kv_cache_precision_b200 import ops
from semantic_aware_adaptive_kv_cache_precision_b200.ops import mixture

pytestmark = pytest.mark.gpu


def draw(*shape, seed=0):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed + sum(shape)),
                       device="cuda")


@pytest.mark.parametrize("M,N,K", [(3, 40, 129), (4, 14400, 65), (5, 9, 128), (16, 33, 260), (17, 700, 64),
                                   (31, 4800, 100), (33, 9600, 33), (100, 4801, 68), (65, 64, 1)])
def test_a_row_of_the_32_bit_product_is_the_same_in_every_tile(M, N, K):
    x, w, bias = draw(M, K), draw(N, K, seed=1), draw(N, seed=2)
    got = ops.linear(x, w, bias)
    want = x.double() @ w.double().T + bias.double()
    bound = 4 * K ** 0.5 * 2.0 ** -24 * float((x.abs().double() @ w.abs().double().T).max()) + 1e-6
    assert float((got.double() - want).abs().max()) <= bound
    for r in {0, M // 2, M - 1}:
        assert torch.equal(ops.linear(x[r:r + 1], w, bias)[0], got[r])
    for rows in (4, 16, 30):
        assert torch.equal(ops.linear(x[:rows], w, bias), got[:rows])


@pytest.mark.parametrize("tokens,outputs,width", [(64, 5, 96), (67, 36, 200), (130, 1, 33), (65, 4, 2048),
                                                  (2501, 5, 96), (701, 36, 200), (8000, 3, 33), (402, 33, 2048)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_router_logits_of_many_tokens_are_those_of_one(tokens, outputs, width, dtype):
    h, w = draw(tokens, width).to(dtype), draw(outputs, width, seed=1)
    got = mixture.router_logits(h, w)
    assert torch.allclose(got.double(), h.double() @ w.double().T, rtol=1e-5, atol=1e-5 * width ** 0.5)
    for t in (0, tokens // 2, tokens - 1):
        assert torch.equal(mixture.router_logits(h[t:t + 1].contiguous(), w)[0], got[t])


@pytest.mark.parametrize("width,group", [(8, 8), (64, 64), (256, 64), (2048, 2048), (2048, 128), (2056, 2056),
                                         (4096, 256), (4096, 4096), (512, 512), (96, 24), (520, 104), (36, 12)])
@pytest.mark.parametrize("gate_silu,gate_first,gated", [(False, False, True), (True, True, True),
                                                        (True, False, True), (False, False, False)])
def test_the_gated_norm_at_every_width(width, group, gate_silu, gate_first, gated):
    tokens, eps, scale = 5, 1e-5, 0.7
    y, w = draw(tokens, width), draw(width, seed=1).to(torch.bfloat16)
    gate = draw(tokens, width + 4, seed=2)[:, :width] if gated else None
    got = ops.norm_gate(y, w, gate, eps, scale, torch.float32, group=group, gate_silu=gate_silu,
                        gate_first=gate_first)
    v, f = y.double(), torch.ones((tokens, width), dtype=torch.float64, device="cuda")
    if gated:
        f = torch.sigmoid(gate.double()) * (gate.double() if gate_silu else 1.0)
    if gate_first:
        v = v * f
    parts = v.view(tokens, width // group, group)
    v = (parts / torch.sqrt((parts * parts).mean(-1, keepdim=True) + eps)).view(tokens, width) * w.double()
    want = (v if gate_first else v * f) * scale
    assert float((got.double() - want).abs().max()) <= 2e-5 * float(want.abs().max())


@pytest.mark.parametrize("tokens,width", [(70, 36), (70, 1024), (70, 2052), (70, 30), (300, 1024), (1100, 260), (150, 2052),
                                          (1100, 262)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rows_gathered_and_summed_at_every_width(tokens, width, dtype):
    experts, top, identity = 5, 3, 2
    h = draw(tokens, width).to(dtype)
    logits = draw(tokens, experts + identity, seed=3)
    r = mixture.route(logits, experts, top, identity)
    rows = mixture.gather_rows(h, r, True)
    products, shared, gate = rows.float() * 2.0, draw(tokens, width, seed=4), draw(tokens, seed=5)
    into = draw(tokens, width, seed=6)
    before = into.double()
    mixture.combine(products, r, False, shared, gate, h, into)
    chosen, weights = r.chosen.long(), r.weights.double()
    want = before + shared.double() * torch.sigmoid(gate.double())[:, None]
    for k in range(top):
        x = h.double() * weights[:, k:k + 1]
        real = (chosen[:, k] < experts)[:, None]
        want = want + torch.where(real, 2.0 * x.to(dtype).double(), x)
    tolerance = 1e-5 if dtype == torch.float32 else 2e-2        # (a weighted row is rounded to its type)
    assert float((into.double() - want).abs().max()) <= tolerance * float(want.abs().max())
    few = mixture.route(logits[:9], experts, top, identity)          # (the same tokens in a short step)
    products = mixture.gather_rows(h[:9], few, True).float() * 2.0
    again = before[:9].float()
    mixture.combine(products, few, False, shared[:9], gate[:9], h[:9], again)
    assert torch.equal(again, into[:9])


@pytest.mark.parametrize("channels,counts", [(520, [300, 1, 2, 3, 5, 90, 4]), (4096, [61, 3, 1, 1]), (1300, [170])])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_the_convolution_of_a_long_step_is_that_of_short_ones(channels, counts, dtype):
    """Sequences begin anywhere among a thread's eight tokens; some have inputs from before the step."""
    tokens, taps = sum(counts), 4
    x, w, b = draw(tokens, channels), draw(channels, taps, seed=1).to(dtype), draw(channels, seed=2).to(dtype)
    before = draw(len(counts), taps - 1, channels, seed=3)

    def conv(rows, counts, state):
        ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
        starts = [sum(counts[:i]) for i in range(len(counts) + 1)]
        step = SimpleNamespace(sequences=len(counts), cu_seqlens=ints(starts), slots=ints(list(range(len(counts)))),
                               token_seq=ints([i for i, c in enumerate(counts) for _ in range(c)]))
        return ops.causal_conv(rows, channels, w, b, state, step, dtype)

    state = before.clone()
    got = conv(x, counts, state)
    at = 0
    for i, n in enumerate(counts):
        alone = before[i:i + 1].clone()
        parts = [conv(x[p:min(p + 33, at + n)], [min(33, at + n - p)], alone) for p in range(at, at + n, 33)]
        assert torch.equal(torch.cat(parts), got[at:at + n]) and torch.equal(alone[0], state[i])
        inputs = torch.cat([before[i], x[at:at + n]]).double()
        sums = sum(inputs[j:j + n] * w[:, j].double() for j in range(taps)) + b.double()
        want = sums * torch.sigmoid(sums)
        off = (got[at:at + n].double() - want).abs() - (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) * want.abs()
        assert float(off.max()) <= 1e-5 * float(want.abs().max())
        at += n
