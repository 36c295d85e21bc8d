"""Host side of the product of a step of few tokens (`csrc/gemm_few.cu`): weights from memory straight
into registers, nothing to set up."""

from __future__ import annotations

import torch

from . import gemm_tc
from ._lib import BF16, call, dtype_code, ptr, sm_count

MAX_TOKENS = 16        # what the kernel takes
ROWS = 16              # weight rows a block


def takes(x: torch.Tensor, weight: torch.Tensor) -> bool:
    """Whether this kernel is the one for the product."""
    return x.shape[0] <= MAX_TOKENS and gemm_tc.takes(x, weight)


def choose_parts(n: int, k: int) -> int:
    """K ranges for blocks of their own whose sums the reader adds: two where the rows alone do not give
    every SM a block and K is long."""
    return 2 if -(-n // ROWS) <= sm_count() and k >= 4096 else 1


def gemm(x: torch.Tensor, weight: torch.Tensor, bias, epi: int, out: torch.Tensor, n: int,
         dual_offset: int = 0, parts: int = 1, clamp: tuple = (0.0, 0.0, 0.0)) -> torch.Tensor:
    """As `gemm_tc.gemm` for up to `MAX_TOKENS` rows of x."""
    m, k = x.shape
    call("sakv_gemm_few", ptr(x), x.stride(0), ptr(weight), m, n, k, parts, epi, dual_offset, ptr(bias),
         dtype_code(bias.dtype) if bias is not None else BF16, ptr(out), out.stride(-2),
         out.stride(0) if parts > 1 else 0, *(float(c) for c in clamp))
    return out
