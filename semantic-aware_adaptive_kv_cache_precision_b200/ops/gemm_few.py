"""Host side of the product of a step of few tokens (`csrc/gemm_few.cu`): every thread its own numbers from
memory to the tensor cores, nothing to set up."""

from __future__ import annotations

import torch

from . import gemm_tc
from ._lib import BF16, call, dtype_code, ptr, sm_count

MAX_TOKENS = 16        # what the kernel takes
ROWS = 16              # weight rows a block
LONGEST_ROW = 3072     # up to this K any number of rows; beyond, what one wave of blocks makes
SHORT_ROW = 2048       # the same for more than 8 tokens
LARGE = 20_000_000     # bytes of a weight, from which on more than 8 tokens go elsewhere


def takes(x: torch.Tensor, weight: torch.Tensor) -> bool:
    """Whether this kernel is the one for the product.

    Its gain is at the ends of a kernel, and it reads x once for every 16 rows of the weight with more
    instructions a byte than `csrc/gemm_tc.cu`, so it is for short rows and for products that one wave of
    blocks makes (by the rows of the weight: a gated product has half as many blocks). Decoded steps after
    1,024 tokens of models of the Qwen2 layout, us, every product by this kernel / by that one, for 1, 8 and
    16 tokens: width 1,024 481 / 737, 587 / 772, 731 / 856; 1,536 924 / 1,083, 1,057 / 1,185, 1,249 / 1,292; 2,048 879 /
    1,080, 1,003 / 1,132, 1,109 / 1,212; 2,560 963 / 1,094, 1,093 / 1,148, 1,284 / 1,241; 3,072 792 / 875, 899 / 931, 1,011
    / 1,005; 3,584 1,289 / 1,261, 1,444 / 1,361, 1,570 / 1,407. With more than 8 tokens x is as much to read as the
    weights (alone, 16 tokens: 46 MB 12.4 / 11.1, 4 MB 2.9 / 3.9; 8 tokens: 10.6 / 10.9, 2.3 / 3.8)."""
    tokens = x.shape[0]
    if tokens > MAX_TOKENS or not gemm_tc.takes(x, weight):
        return False
    n, k = weight.shape
    if tokens > 8 and n * k * weight.element_size() > LARGE:
        return False
    return k <= (LONGEST_ROW if tokens <= 8 else SHORT_ROW) or n <= ROWS * sm_count()


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
