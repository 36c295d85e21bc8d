"""Host side of the product of a step of few tokens (`csrc/gemm_few.cu`): weights from memory straight
into registers, nothing to set up."""

from __future__ import annotations

import torch

from . import gemm_tc
from ._lib import BF16, call, dtype_code, ptr, sm_count

MAX_TOKENS = 16        # what the kernel takes
ROWS = 16              # weight rows a block
SHORT_ROW = 2048       # up to this K any number of rows; beyond, what one wave of blocks makes
LARGE = 20_000_000     # bytes of a weight, from which on more than 8 tokens go elsewhere


def takes(x: torch.Tensor, weight: torch.Tensor) -> bool:
    """Whether this kernel is the one for the product.

    Its gain is at the ends of a kernel, and it reads x once for every 16 rows of the weight with more
    instructions a byte than `csrc/gemm_tc.cu`, so it is for short rows and for products that one wave of
    blocks makes. Decode steps, us (this kernel for every product / that one): width 1,536, one user 955 /
    1,101 and 8 users 1,095 / 1,254; width 1,024 and 4 users 425 / 481. Width 3,584 and 8 users, rows of 3,584 in
    more than a wave: alone the products are as fast (44 / 43), but in the steps after a prompt of 9,216
    tokens, whose power holds the clocks down (every kernel of a step takes 1.7 times what it does after
    2,560), instructions are what bounds this one and a step takes 6,831 / 3,401. With more than 8 tokens x
    is as much to read as the weights, and a large product takes longer (46 MB, 16 tokens: 14.9 / 11.3; 4
    MB: 3.1 / 3.4; a step of 16 users 692 / 680, with the limit 688)."""
    tokens = x.shape[0]
    if tokens > MAX_TOKENS or not gemm_tc.takes(x, weight):
        return False
    n, k = weight.shape
    if tokens > 8 and n * k * weight.element_size() > LARGE:
        return False
    return k <= SHORT_ROW or n <= ROWS * sm_count()


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
