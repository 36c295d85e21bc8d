"""The forms of the small kernels that go by groups of four numbers, at the widths where their number of
groups a thread changes, against the same in 64 bits."""

from __future__ import annotations

from types import SimpleNamespace

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


@pytest.mark.parametrize("width", [4, 1020, 1024, 1028, 2048, 2052, 4096, 4100])
@pytest.mark.parametrize("streams", [1, 2, 4])
def test_streams_between_two_sublayers(streams, width):
    g = torch.Generator(device=DEV).manual_seed(width + streams)
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)
    n, eps = 3, 1e-5
    xs, y = rand(streams, n, width), rand(n, width)
    mix, out_w, in_w = rand(streams, streams).to(BF), rand(streams).to(BF), rand(streams).to(BF)
    norm_w, blend = (1 + 0.1 * rand(width)).to(BF), torch.rand(width, generator=g, device=DEV).to(BF)
    kept = rand(5, width)
    step = SimpleNamespace(sequences=n, token_seq=torch.arange(n, dtype=torch.int32, device=DEV),
                           slots=torch.tensor([4, 0, 2], dtype=torch.int32, device=DEV))
    want = torch.einsum("st,snw->tnw", mix.double(), xs.double()) + out_w.double()[:, None, None] * y.double()
    low = rms(torch.einsum("s,snw->nw", in_w.double(), want), eps) * norm_w.double()
    got, state = xs.clone(), kept.clone()
    out = ops.streams_step(got, y=y, mix=mix, out_w=out_w, in_w=in_w, norm_w=norm_w, eps=eps, out_dtype=BF,
                           shift=(state, blend, step))
    near(got, want, 32)
    near(state[[4, 0, 2]], low, 32)
    assert torch.equal(state[[1, 3]], kept[[1, 3]])
    near(out, low + (kept[[4, 0, 2]].double() - low) * blend.double())
    again = xs.clone()
    near(ops.streams_step(again, in_w=in_w, norm_w=norm_w, eps=eps),
         rms(torch.einsum("s,snw->nw", in_w.double(), xs.double()), eps) * norm_w.double(), 32)
    assert torch.equal(again, xs)
    assert ops.streams_step(again, y=y, mix=mix, out_w=out_w, reduce=False) is None
    near(again, want, 32)


@pytest.mark.parametrize("width", [4, 1024, 1028, 2048, 2052, 4096, 4100])
def test_layer_norm_of_a_sublayer_s_output_and_of_the_stream(width):
    g = torch.Generator(device=DEV).manual_seed(width)
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)
    n, eps = 4, 1e-5
    x, y = rand(n, width) + 0.5, 3 * rand(n, width) - 1
    w_after, w = ((1 + 0.2 * rand(width)).to(BF) for _ in range(2))

    def norm(a):
        d = a - a.mean(-1, keepdim=True)
        return d / (d.square().mean(-1, keepdim=True) + eps).sqrt()

    stream = x.clone()
    out = ops.layer_norm(stream, w, eps, BF, add=y, add_weight=w_after)
    want = x.double() + norm(y.double()) * w_after.double()
    near(stream, want, 32)
    near(out, norm(want) * w.double())
    rows = torch.tensor([3, 0, 3], dtype=torch.int32, device=DEV)
    near(ops.layer_norm(x, w, eps, torch.float32, rows=rows), (norm(x.double()) * w.double())[rows.long()], 32)
    stream = x.clone()
    assert ops.layer_norm(stream, None, eps, BF, add=y, add_weight=w_after) is None
    near(stream, want, 32)


@pytest.mark.parametrize("q_rank,rank,rot", [(4, 8, 4), (512, 516, 64), (1024, 512, 8), (1536, 512, 64),
                                             (2048, 2044, 512), (4096, 256, 64), (4100, 64, 64), (0, 1024, 4)])
@pytest.mark.parametrize("write", [True, False])
def test_latents_of_a_step(q_rank, rank, rot, write):
    g = torch.Generator(device=DEV).manual_seed(q_rank + rank)
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)
    T, eps = 4, 1e-5
    down = 2 * rand(T, q_rank + rank + rot)
    wq, wk = ((1 + 0.2 * rand(max(n, 1))).to(BF) for n in (q_rank, rank))
    angle = 6 * torch.rand(64, rot // 2, generator=g, device=DEV)
    step = SimpleNamespace(positions=torch.tensor([0, 9, 63, 1], dtype=torch.int32, device=DEV),
                           token_seq=torch.tensor([0, 0, 0, 1], dtype=torch.int32, device=DEV))
    view = SimpleNamespace(keys=torch.zeros(2, 1, 64, rank + rot, dtype=BF, device=DEV),
                           block_table=torch.tensor([[1], [0]], dtype=torch.int32, device=DEV))
    got = ops.latent_prepare(down, q_rank, rank, rot, wq if q_rank else None, wk, eps, step, view, angle.cos(),
                             angle.sin(), BF, write_cache=write, interleaved=True)
    d = down.double()
    if q_rank:
        near(got, rms(d[:, :q_rank], eps) * wq.double())
    at = step.positions.long()
    c, s = (t[at].double() for t in (angle.cos(), angle.sin()))
    a, b = d[:, q_rank + rank::2], d[:, q_rank + rank + 1::2]
    turned = torch.stack([a * c - b * s, b * c + a * s], -1).view(T, rot)
    want = torch.cat([rms(d[:, q_rank:q_rank + rank], eps) * wk.double(), turned], 1)
    stored = view.keys[view.block_table[step.token_seq.long(), 0].long(), 0, at]
    if write:
        near(stored, want)
    else:
        assert (view.keys == 0).all()


@pytest.mark.parametrize("n_state", [4, 16, 128])
@pytest.mark.parametrize("rank", [8, 16, 40, 136, 256, 264, 7])
def test_step_sizes_made_inside_a_decoded_step(n_state, rank):
    """A channel's lanes share out the products of its step size, eight columns at a time (a rank that is
    no multiple of eight: one after another): the outputs of the steps made before, in 64 bits."""
    g = torch.Generator(device=DEV).manual_seed(rank + n_state)
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)
    T, channels = 3, 132
    x, z = rand(T, channels).to(BF), rand(T, channels)
    columns = -(-(rank + 2 * n_state) // 4) * 4
    low = 0.3 * rand(T, columns)
    w, b = (0.1 * rand(channels, rank)).to(BF), (rand(channels) - 1).to(BF)
    a_log, skip = (0.5 * rand(channels, n_state)).to(BF), rand(channels).to(BF)
    state = rand(T, channels, n_state)
    step = SimpleNamespace(sequences=T, max_new=1, is_decode=True,
                           cu_seqlens=torch.arange(T + 1, dtype=torch.int32, device=DEV),
                           slots=torch.arange(T, dtype=torch.int32, device=DEV))
    dt = torch.nn.functional.softplus(low[:, :rank].double() @ w.double().T + b.double())
    B, C = low[:, rank:rank + n_state].double(), low[:, rank + n_state:rank + 2 * n_state].double()
    S = torch.exp(-dt[..., None] * torch.exp(a_log.double())) * state.double() + \
        (dt * x.double())[..., None] * B[:, None]
    want = (torch.einsum("tcn,tn->tc", S, C) + skip.double() * x.double()) * torch.nn.functional.silu(z.double())
    got = ops.selective_scan(x, None, low, rank, rank + n_state, n_state, z, a_log, skip, state, step,
                             dt_weight=w, dt_bias=b)
    near(state, S, 32)
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * want.abs().max()).all()
