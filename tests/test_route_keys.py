"""Which experts a token gets (`csrc/moe.cu`): the largest ranks in order, ties to the lowest index, never one
that is not a number, at the sizes where a lane's ranks begin to take another register or leave them."""

import math

import pytest
import torch

from semantic_aware_adaptive_kv_cache_precision_b200.ops import mixture

pytestmark = pytest.mark.gpu


def chosen(ranks, top):
    order = sorted((i for i, v in enumerate(ranks) if not math.isnan(v)), key=lambda i: (-ranks[i], i))
    return [order[k] if k < len(order) else k for k in range(top)]


@pytest.mark.parametrize("tokens", [1, 9, 40, 700])
@pytest.mark.parametrize("experts", [1, 31, 32, 33, 64, 127, 128, 129, 200])
@pytest.mark.parametrize("biased", [False, True])
def test_the_largest_in_order(tokens, experts, biased):
    g = torch.Generator().manual_seed(tokens + experts)
    top = min(experts, 12)
    values = torch.randint(-6, 7, (tokens, experts), generator=g).float() / 4          # many ties
    values[values == 0.25] = -0.0
    if biased:              # a logit of 0 is a score of one half, exactly
        logits, bias = torch.zeros(tokens, experts), values[0].clone()
        ranks = (bias + 0.5).expand(tokens, experts)
    else:
        logits, bias = values, None
        logits[0, : max(1, experts // 2)] = float("nan")
        logits[-1, experts // 2:] = float("-inf")
        ranks = logits
    r = mixture.route(logits.cuda(), experts, top, bias=None if bias is None else bias.cuda())
    got = r.chosen.cpu().tolist()
    for t in {0, tokens // 2, tokens - 1}:
        assert got[t] == chosen(ranks[t].tolist(), top)
