"""Cached attention in bfloat16 on the tensor cores (`csrc/attention_mma.cu`): which calls it
takes, and its launch."""

from __future__ import annotations

import torch

from . import _lib
from ._lib import call, ptr

#: (key columns, value columns, values inside the key rows, most maps a head) of the compiled kernels
SHAPES = {(64, 64, False): 1, (128, 128, False): 2, (128, 256, False): 2, (576, 512, True): 1}


def takes(q: torch.Tensor, head_stride: int, k_cache: torch.Tensor, v_cache, dim: int, vdim: int,
          maps: int = 1, q2=None, q_split: int = 0) -> bool:
    """Whether the tensor-core kernel takes the call: bfloat16, one of the compiled pairs of
    widths, and every row of queries, keys and values beginning at a multiple of 16 bytes (they are
    copied in pieces of 16). Against the kernel that scores a key a lane, us, 16 heads over latent rows
    and 8 heads of 2 at 128 columns: a prompt of 3,001 tokens 14,597 -> 1,131 and 2,587 -> 244; 8 decoded
    tokens of 2,048 keys 132 -> 37 and 74 -> 39; the steps that mix both in `csrc/attention_mma.cu`. Of 150
    calls from one token on it is slower only where a block's rows are nearly all empty: prompts of 16
    tokens with a head a key/value head 8 -> 11 (they stay here: a prompt's result must not depend
    on how it is cut)."""
    if q.dtype != torch.bfloat16 or SHAPES.get((dim, vdim, v_cache is None), 0) < maps:
        return False
    rows = [(q, q.stride(0), head_stride), (k_cache, k_cache.shape[3], 0)]
    if v_cache is not None:
        rows.append((v_cache, v_cache.shape[3], 0))
    if q2 is not None:
        rows.append((q2, q2.stride(0), q2.stride(1) | q_split))
    return all(t.data_ptr() % 16 == 0 and a % 8 == 0 and b % 8 == 0 for t, a, b in rows)


def attention(q, head_stride, k_cache, v_cache, positions, token_seq, block_table, heads, dim, vdim,
              scale, *, maps=1, q2=None, q_split=0, window=None, chunk=None, keep_first=0, slope=None,
              rate=None, softcap=None, linear=None, sink=None, head_gate=None, elem_gate=None,
              map_gate_off=None, lam=0.0, out_scale=1.0, eps=0.0, decode=False, key_splits=1,
              ordered=True, cu_seqlens=None):
    """The arguments as `ops.cached_attention` and `ops.distance_attention` have checked them.
    `decode`: a block (and `key_splits` of them) takes one token; else 64 rows of a prompt, of one
    sequence with `cu_seqlens` (int32 [sequences + 1]: where every sequence's tokens begin), of one
    run of consecutive tokens without. `ordered`: the kernels begin when the one before them has
    ended (False: overlapped with it, for a caller whose neighbours are this library's own
    kernels)."""
    tokens = q.shape[0]
    out = torch.empty((tokens, heads * vdim), dtype=q.dtype, device=q.device)
    if not decode:
        key_splits = 1
    sums = stats = None
    if decode and (maps == 2 or key_splits > 1):
        rows = key_splits * tokens * heads * maps
        sums = torch.empty((rows, vdim), dtype=torch.float32, device=q.device)
        stats = torch.empty((rows, 2), dtype=torch.float32, device=q.device)
    if maps == 1:
        map_gate_off = None
    call("sakv_attention_mma", ptr(q), q.stride(0), head_stride, ptr(q2),
         0 if q2 is None else q2.stride(0), 0 if q2 is None else q2.stride(1), q_split, ptr(out),
         ptr(k_cache), k_cache.shape[3], ptr(v_cache), 0 if v_cache is None else v_cache.shape[3],
         ptr(positions), ptr(token_seq), ptr(cu_seqlens), block_table.shape[0], ptr(block_table),
         block_table.shape[1], tokens, heads,
         k_cache.shape[1], maps, dim, vdim, float(scale), int(window) if window else 0,
         int(chunk) if chunk else 0, int(keep_first), ptr(slope), ptr(rate), float(softcap or 0.0),
         ptr(linear), ptr(sink), ptr(head_gate), 0 if head_gate is None else head_gate.stride(0),
         ptr(elem_gate), 0 if elem_gate is None else elem_gate.stride(0),
         None if map_gate_off is None else q.data_ptr() + 2 * map_gate_off, q.stride(0),
         float(out_scale), float(lam), float(eps), int(decode), int(key_splits), ptr(sums), ptr(stats),
         int(ordered))
    if sums is not None and tokens:
        _lib.launches += 1          # the call launched the fold kernel too
    return out
