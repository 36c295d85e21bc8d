"""The product of a step of few tokens (csrc/gemm_few.cu) against the same sums in 64 bits: token counts
on both sides of a group of eight, rows and columns that end inside a block's 16 and a group of 32,
columns beyond what a warp asks for at once, every epilogue, ranges of K left apart."""

from __future__ import annotations

import pytest
import torch

from semantic_aware_adaptive_kv_cache_precision_b200 import ops
from semantic_aware_adaptive_kv_cache_precision_b200.ops import gemm_few, gemm_tc

pytestmark = pytest.mark.gpu

DEV = "cuda"


def operands(m, n, k, seed=0):
    g = torch.Generator(device=DEV).manual_seed(1000 * m + n + k + seed)
    x = torch.randn((m, k + 8), generator=g, device=DEV).bfloat16()[:, :k]      # wider rows
    w = (torch.randn((n, k), generator=g, device=DEV) * k ** -0.5).bfloat16()
    return x, w, g


def close(got, want, bits, k):
    # exact products summed in fp32: a warp's sum (of about 1, as the whole) passes k / 128 products of the
    # tensor cores, each of which may cut a unit of its last place, 2^-23, and eight such sums are added;
    # 16-bit results are rounded once more, by half a unit of 2^-8
    tol = 2.0 ** -8 * want.abs() if bits == 16 else 0.0
    assert ((got.double() - want).abs() <= tol + (16 + k / 128) * 2.0 ** -23 * (1 + want.abs())).all()


@pytest.mark.parametrize("m", [1, 2, 7, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(1, 8), (15, 24), (16, 32), (17, 264), (100, 1536), (40, 3080), (33, 8960)])
def test_every_epilogue_at_edges(m, n, k):
    x, w, g = operands(m, n, k)
    want = x.double() @ w.double().T
    bias = torch.randn(n, generator=g, device=DEV)
    out = torch.empty((m, n), device=DEV)
    close(gemm_few.gemm(x, w, bias, gemm_tc.EPI_F32, out, n), want + bias.double(), 32, k)
    b16 = bias.bfloat16()
    out16 = torch.empty((m, n), dtype=torch.bfloat16, device=DEV)
    close(gemm_few.gemm(x, w, b16, gemm_tc.EPI_BF16, out16, n), want + b16.double(), 16, k)
    stream = torch.randn((m, n), generator=g, device=DEV)
    before = stream.double()
    close(gemm_few.gemm(x, w, None, gemm_tc.EPI_ACCUM, stream, n), before + want, 32, k)
    close(gemm_few.gemm(x, w, None, gemm_tc.EPI_RELU2, out16, n), want.clamp_min(0) ** 2, 16, k)
    up = (torch.randn((n, k), generator=g, device=DEV) * k ** -0.5).bfloat16()
    both = torch.cat([w, up])
    u = x.double() @ up.double().T
    close(gemm_few.gemm(x, both, None, gemm_tc.EPI_GATED, out16, n, dual_offset=n),
          torch.nn.functional.silu(want) * u, 16, k)
    limit, alpha, plus = 0.7, 1.702, 1.0
    a, b = want.clamp_max(limit), u.clamp(-limit, limit)
    close(gemm_few.gemm(x, both, None, gemm_tc.EPI_CLAMPED, out16, n, dual_offset=n,
                        clamp=(limit, alpha, plus)), a * torch.sigmoid(alpha * a) * (b + plus), 16, k)
    for parts in (2, 3):
        sums = torch.empty((parts, m, n), device=DEV)
        gemm_few.gemm(x, w, bias, gemm_tc.EPI_F32, sums, n, parts=parts)
        close(sums.sum(0), want + bias.double(), 32, k)


def test_a_row_does_not_feel_values_beyond_its_own():
    """Infinities in the columns behind a row's end, in other tokens' rows and in rows of the weight that
    are not asked for."""
    x, w, _ = operands(3, 20, 40)
    whole = torch.full((5, 48), float("inf"), dtype=torch.bfloat16, device=DEV)
    whole[:3, :40] = x
    rows = torch.full((30, 40), float("inf"), dtype=torch.bfloat16, device=DEV)
    rows[:20] = w
    out = torch.empty((3, 20), device=DEV)
    close(gemm_few.gemm(whole[:3, :40], rows[:20], None, gemm_tc.EPI_F32, out, 20),
          x.double() @ w.double().T, 32, 40)


def test_the_rule_and_the_ops_that_follow_it():
    """`linear`, `gated_up` and `dense_up` give the same on both sides of the rule's last token."""
    for m in (gemm_few.MAX_TOKENS, gemm_few.MAX_TOKENS + 1):
        x, w, g = operands(m, 256, 512)
        x = x.contiguous()
        assert gemm_few.takes(x, w) == (m <= gemm_few.MAX_TOKENS)
        want = x.double() @ w.double().T
        close(ops.linear(x, w, out_dtype=torch.float32), want, 32, 512)
        close(ops.linear(x, w), want, 16, 512)
        close(ops.dense_up(x, w), want.clamp_min(0) ** 2, 16, 512)
        close(ops.gated_up(x, w), torch.nn.functional.silu(want[:, :128]) * want[:, 128:], 16, 512)
        stream = torch.zeros((m, 256), device=DEV)
        close(ops.linear(x, w, accumulate_into=stream), want, 32, 512)
    x, w, _ = operands(4, 64, 8192)
    stream = torch.ones((4, 64), device=DEV)
    left = ops.linear(x, w, accumulate_into=stream, may_defer=True)
    assert isinstance(left, ops.Deferred) and left.delta.shape == (2, 4, 64)
    close(left.delta.sum(0), x.double() @ w.double().T, 32, 8192)
    assert (stream == 1).all()


@pytest.mark.parametrize("m,k,taken", [(1, 3072, True), (8, 3072, True), (8, 3080, False), (9, 2048, True),
                                       (9, 2056, False), (16, 2048, True), (17, 1024, False)])
def test_the_rule_s_lines(m, k, taken):
    """By tokens and columns where the rows are more than a wave of blocks makes; any columns up to there."""
    wave = gemm_few.ROWS * ops.sm_count()
    x = torch.zeros((m, k), dtype=torch.bfloat16, device=DEV)
    w = torch.zeros((wave + 16, k), dtype=torch.bfloat16, device=DEV)
    assert gemm_few.takes(x, w) == taken
    assert gemm_few.takes(x, w[:wave]) == (m <= gemm_few.MAX_TOKENS)
    large = torch.zeros((gemm_few.LARGE // (2 * k) + 1, k), dtype=torch.bfloat16, device=DEV)
    assert gemm_few.takes(x, large) == (taken and m <= 8)
