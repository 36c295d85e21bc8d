"""The forms of the small kernels that go by groups of four numbers, at the widths where their number of
groups a thread changes, against the same in 64 bits."""

from __future__ import annotations

import pytest
import torch

from semantic_aware_adaptive_kv_cache_precision_b200 import ops

pytestmark = pytest.mark.gpu

DEV, BF = "cuda", torch.bfloat16


def near(got, want, bits=16):
    """A few units of the last place of a sum of a few thousand squares in fp32, and half a unit of the
    result's type."""
    unit = 2.0 ** -8 if bits == 16 else 2.0 ** -22
    assert ((got.double() - want).abs() <= unit * want.abs() + 2.0 ** -20 * want.abs().max()).all()


def kernels_of(run):
    """The names of the kernels that `run` launches, and its result."""
    from torch.profiler import ProfilerActivity, profile
    run()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        out = run()
        torch.cuda.synchronize()
    return " ".join(e.name for e in prof.events()), out


def rms(x, eps):
    return x / (x.square().mean(-1, keepdim=True) + eps).sqrt()


@pytest.mark.parametrize("norm,weights", [("whole", True), ("head", True), ("head", False), (None, False)])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,rot", [
    (1, 1, 4, 4, 0), (8, 2, 128, 128, 128), (9, 3, 112, 44, 16), (16, 4, 128, 64, 64), (32, 8, 64, 128, 32),
    (33, 1, 32, 2048, 8), (32, 4, 128, 72, 128)])
def test_queries_keys_and_values_of_a_step(norm, weights, heads, kv_heads, dim, vdim, rot):
    """Widths of one, two and four groups a thread with one norm over all heads, several blocks of one group
    without; offsets of whole fours. (Norms a head of 112 columns go by the general kernel.)"""
    g = torch.Generator(device=DEV).manual_seed(heads + dim)
    T, eps, off = 5, 1e-5, 8
    qc, kc, vc = heads * dim, kv_heads * dim, kv_heads * vdim
    proj = torch.randn(T, off + qc + kc + vc + 4, generator=g, device=DEV)
    wq = wk = None
    if weights:
        wq, wk = ((1 + 0.3 * torch.randn(n, generator=g, device=DEV)).to(BF)
                  for n in ((qc, kc) if norm == "whole" else (dim, dim)))
    angle = torch.rand(64, rot // 2, generator=g, device=DEV) * 6
    cos, sin = (angle.cos(), angle.sin()) if rot else (None, None)
    positions = torch.tensor([0, 1, 17, 63, 5], dtype=torch.int32, device=DEV)
    seq = torch.tensor([0, 0, 0, 0, 1], dtype=torch.int32, device=DEV)
    table = torch.tensor([[1], [0]], dtype=torch.int32, device=DEV)
    temp = torch.rand(64, generator=g, device=DEV) + 0.5
    keys = torch.zeros(2, kv_heads, 64, dim, dtype=BF, device=DEV)
    values = torch.zeros(2, kv_heads, 64, vdim, dtype=BF, device=DEV)
    names, got = kernels_of(lambda: ops.qk_prepare(
        proj, off, off + qc, off + qc + kc, heads, kv_heads, dim, vdim, wq, wk, eps, cos, sin, positions, seq,
        table, keys, values, BF, norm=norm, temperature=temp))
    assert ("qk_prepare_vec_kernel" in names) == (norm != "head" or dim & (dim - 1) == 0), names

    def shaped(x, w, n):
        if norm == "whole":
            x = rms(x, eps) * (1.0 if w is None else w.double())
        x = x.view(T, n, dim)
        if norm == "head":
            x = rms(x, eps) * (1.0 if w is None else w.double())
        if rot:
            c, s = (t[positions.long()].double()[:, None] for t in (cos, sin))
            a, b = x[..., :rot // 2], x[..., rot // 2:rot]
            x = torch.cat([a * c - b * s, b * c + a * s, x[..., rot:]], -1)
        return x

    p = proj.double()
    near(got.view(T, heads, dim), shaped(p[:, off:off + qc], wq, heads) * temp[positions.long()].double()[:, None, None])
    k, v = shaped(p[:, off + qc:off + qc + kc], wk, kv_heads), p[:, off + qc + kc:off + qc + kc + vc].view(T, kv_heads, vdim)
    block = table[seq.long(), 0].long()
    near(keys[block, :, positions.long()], k)
    near(values[block, :, positions.long()], v)
    kept = torch.ones(2, 64, dtype=torch.bool, device=DEV)
    kept[block, positions.long()] = False
    assert (keys.transpose(1, 2)[kept] == 0).all() and (values.transpose(1, 2)[kept] == 0).all()
