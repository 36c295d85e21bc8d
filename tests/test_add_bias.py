"""The bias of a prompt's fp32 product (`csrc/elementwise.cu`): one addition an element, the same bits (but for a
-0 that a bias of zero is not added to)."""

import pytest
import torch

from semantic_aware_adaptive_kv_cache_precision_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [65, 130, 1025])
@pytest.mark.parametrize("n", [8, 1000, 1032])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shift", [0, 1])
def test_it_is_the_addition(tokens, n, dtype, shift):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(tokens, 64, generator=g, device="cuda").bfloat16()
    w = torch.randn(n + 3, 64, generator=g, device="cuda").bfloat16()[:n + (3 if shift else 0)].contiguous()
    bias = torch.randn(w.shape[0] + shift, generator=g, device="cuda").to(dtype)[shift:]
    bias[n // 2:] = 0
    want = ops.linear(x, w, out_dtype=torch.float32) + bias.float()
    assert torch.equal(ops.linear(x, w, bias, out_dtype=torch.float32), want)
    into = torch.zeros_like(want)
    assert torch.equal(ops.linear(x, w, bias, accumulate_into=into), want)
