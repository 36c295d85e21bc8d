"""The grouped products of a mixture on tcgen05 (`csrc/moe_tc.cu`): the rules that choose it and its
tiles (no GPU needed), and its results at the edges of tiles, with experts that nobody chose."""

import pytest
import torch

from semantic_aware_adaptive_kv_cache_precision_b200.ops import mixture
from semantic_aware_adaptive_kv_cache_precision_b200.ops._lib import call, ptr


def test_the_rules_of_the_tiles():
    def asks(dtype=torch.bfloat16, n=64, k=64, offset=0, two=True):
        rows = torch.zeros(4 * k + 8, dtype=dtype)[offset:][:4 * k].view(4, k)
        w = torch.zeros((3, n, k), dtype=dtype)
        return mixture.tc_takes(rows, w, w if two else None)

    assert asks() and asks(two=False) and asks(n=8, k=8) and asks(offset=8)
    assert not asks(dtype=torch.float32) and not asks(n=12) and not asks(k=12) and not asks(offset=4)
    assert mixture.few_tiles(4, 32, 1024, True) and not mixture.few_tiles(32, 16, 1024, True)
    assert not mixture.few_tiles(6000, 2, 1024, False)


@pytest.mark.parametrize("rows,experts,n,k,dual,faster", [
    (2, 16, 64, 48, False, "tile"), (4000, 4, 48, 64, True, "tile"), (32, 16, 1024, 512, False, "tile"),
    (8000, 32, 64, 48, False, "tile"), (8, 8, 256, 256, True, "tile"), (128, 2, 1024, 1024, False, "few"),
    (2, 16, 1024, 1024, True, "few"), (8, 4, 1024, 2048, True, "few"), (400, 4, 1024, 1024, True, "large"),
    (1200, 4, 1024, 1024, False, "large"), (8000, 32, 2048, 1024, False, "large")])
def test_a_product_takes_the_form_that_was_measured_to_be_the_fastest(rows, experts, n, k, dual, faster):
    assert mixture.tc_faster(rows, experts, n, k, dual) == (faster != "tile")
    if faster != "tile":
        assert mixture.few_tiles(rows, experts, n, dual, k) == (faster == "few")


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,experts,top,width,ff", [(1, 4, 2, 64, 48), (33, 16, 2, 256, 256), (70, 4, 2, 1024, 512)])
def test_a_grouped_product_is_the_same_in_every_form(tokens, experts, top, width, ff, monkeypatch):
    """bfloat16 products are exact in fp32; the sums may be taken in another order (2^-24 a term)."""
    g = torch.Generator(device="cuda").manual_seed(tokens)

    def draw(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    r = mixture.route(draw(tokens, experts), experts, top)
    rows = mixture.gather_rows(draw(tokens, width).to(torch.bfloat16), r, False)
    gate, up = draw(experts, ff, width).to(torch.bfloat16), draw(experts, ff, width).to(torch.bfloat16)
    got = {}
    for form in ("tile", "few", "large"):
        with monkeypatch.context() as m:
            m.setattr(mixture, "tc_faster", lambda *a: form != "tile")
            m.setattr(mixture, "few_tiles", lambda *a: form == "few")
            got[form] = (mixture.grouped_product(rows, r, gate, None),
                         mixture.grouped_product(rows, r, gate, up, 30.0, 1.5).float())
    bound = 4 * width ** 0.5 * 2.0 ** -24 * float((rows.float().abs() @ gate.float().abs().amax(0).T).max())
    for form in ("few", "large"):
        assert float((got[form][0] - got["tile"][0]).abs().max()) <= bound
        off = (got[form][1] - got["tile"][1]).abs() - 2.0 ** -7 * got["tile"][1].abs()
        assert float(off.max()) <= 100 * bound                  # (times the other factor, at most 31)


@pytest.mark.gpu
@pytest.mark.parametrize("few", [True, False])
@pytest.mark.parametrize("n,k", [(8, 8), (64, 72), (136, 200), (264, 1032)])
@pytest.mark.parametrize("counts", [(1,), (0, 31, 32, 33, 0), (127, 0, 0, 128, 129, 1), (0, 0, 300)])
def test_products_at_the_edges_of_tiles(counts, n, k, few):
    """Against float64. A gated output is rounded to bfloat16 once (2^-8 of it) and its activation
    taken with the hardware's exponential and division (some 2^-20); sums of k products are fp32."""
    g = torch.Generator(device="cuda").manual_seed(n + k + len(counts))

    def draw(*shape):
        return torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)

    total, experts = sum(counts), len(counts)
    rows, gate, up = draw(total + 3, k), draw(experts, n, k), draw(experts, n, k)   # (3 rows of nobody)
    offsets = torch.tensor([sum(counts[:i]) for i in range(experts + 1)], dtype=torch.int32, device="cuda")
    plain = torch.full((total + 3, n), 7.0, dtype=torch.float32, device="cuda")
    gated = torch.full((total + 3, n), 7.0, dtype=torch.bfloat16, device="cuda")
    limit, alpha, plus = 20.0, 1.25, 0.5
    call("sakv_moe_tc", ptr(rows), total + 3, ptr(gate), None, ptr(offsets), experts, ptr(plain), n, k,
         0.0, 0.0, 0.0, int(few))
    call("sakv_moe_tc", ptr(rows), total + 3, ptr(gate), ptr(up), ptr(offsets), experts, ptr(gated), n, k,
         limit, alpha, plus, int(few))
    assert bool((plain[total:] == 7).all()) and bool((gated[total:] == 7).all())
    for e in range(experts):
        lo, hi = int(offsets[e]), int(offsets[e + 1])
        if lo == hi:
            continue
        x = rows[lo:hi].double()
        a, b = x @ gate[e].double().T, x @ up[e].double().T
        size = x.abs() @ gate[e].double().abs().T
        assert bool(((plain[lo:hi].double() - a).abs() <= 4 * k ** 0.5 * 2.0 ** -24 * size.max()).all())
        c, d = a.clamp(max=limit), b.clamp(-limit, limit)
        want = c * torch.sigmoid(alpha * c) * (d + plus)
        off = (gated[lo:hi].double() - want).abs()
        assert bool((off <= 2.0 ** -8 * want.abs() + 1e-4 * want.abs().max()).all())


@pytest.mark.gpu
@pytest.mark.parametrize("few", [True, False])
def test_the_gated_activation_far_out(few):
    """g sigmoid(alpha g) where 1 + exp(-alpha g) lies above 2^126: a quotient by an approximate
    reciprocal is 0 there, the number itself is a normal one."""
    rows = torch.zeros((3, 8), dtype=torch.bfloat16, device="cuda")
    rows[:, 0] = torch.tensor([-70.0, -69.5, 1.0])
    gate = torch.zeros((1, 8, 8), dtype=torch.bfloat16, device="cuda")
    gate[0, :, 0] = 1.0
    up = torch.zeros_like(gate)
    offsets = torch.tensor([0, 3], dtype=torch.int32, device="cuda")
    out = torch.zeros((3, 8), dtype=torch.bfloat16, device="cuda")
    call("sakv_moe_tc", ptr(rows), 3, ptr(gate), ptr(up), ptr(offsets), 1, ptr(out), 8, 8, 100.0, 1.2525, 1.0,
         int(few))
    x = rows[:, :1].double().expand(3, 8)
    want = x * torch.sigmoid(1.2525 * x)
    assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs()).all())
