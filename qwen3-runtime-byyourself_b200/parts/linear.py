"""y = x . W^T for weights stored [out, in], the one matrix product of the model.

32-bit operands go to the library's own fmaf kernel (true 32-bit, fixed summation
order).  bfloat16 operands go to the library's own tensor-core kernels: to its
weight-streaming kernel for the few rows of a decode step and to its TMA + tcgen05
kernels beyond (weights first with K split over a cluster for up to a few hundred rows,
tokens first and persistent on pairs of SMs for prompts); widths that are no multiple of 8 go to a CUDA-core kernel
with 32-bit accumulation.  No product goes to a library, where the reference's engine
calls cublasGemmEx for every projection (src/ops/linear.cpp:165-193: bfloat16 in, 32-bit
accumulate).  Another kernel can be registered for a shape (`set_bf16_kernel`).
"""
from __future__ import annotations

import functools
from typing import Callable, Optional

import torch

from ..csrc import ops

_bf16_kernel: Optional[Callable] = None
skinny_rows = 8      # up to this many rows the weight-streaming kernel runs


def set_bf16_kernel(fn: Optional[Callable]) -> None:
    """`fn(x, w, out) -> bool` may take a bfloat16 product; False hands it to the kernels below."""
    global _bf16_kernel
    _bf16_kernel = fn


def set_bf16_kernel_active() -> bool:
    """Whether another kernel has been registered for bfloat16 products (fused projections then stand back)."""
    return _bf16_kernel is not None


# Microseconds per 64-wide K step of a tile and per block for its start and end, measured on B200 (the unsplit pairs form
# gives its own estimate, of the tiles it would take).
_STEP_US = {"pair": 0.33, "prompt128": 0.29, "weights_first": 0.40}
_BLOCK_US = {"prompt128": 4.0}
# A tile with K split over the pairs of a cluster is not persistent: every wave pays the start of the stream and the
# meeting of the partial tiles over distributed shared memory, and the launch a little more.  (K 4,096 and 12,288: two ranges
# 18.3 and 39.7 us, three 16.2 and 29.5; the weights-first form with a range per block of a cluster 13.4 and 26.4 with four, 19.7 with two,
# whose blocks have twice as many tokens to add up and write.)  With K up to 2,048 these decide: 300 tokens of 4,096 x 2,048 in 32 bits weights
# first 16.4, single SMs 11.0, pairs with two ranges 14.2; 600 tokens of 2,048 x 1,024 pairs 8.7, single SMs 6.2; 256 tokens of 3,072 x 4,096
# weights first in four ranges 14.9, pairs in four 15.6, single SMs 16.6; 600 of them 21.9 (two ranges) against 20.2 on pairs without a split.
_PAIR_SPLIT_WAVE_US, _PAIR_SPLIT_LAUNCH_US = 6.0, 2.5
_WEIGHTS_FIRST_US = {1: 5.0, 2: 9.0, 4: 7.0, 8: 7.0}      # a block's start and end, by the ranges of K


@functools.lru_cache(maxsize=4096)
def pair_plan(M: int, N: int, K: int, may_row: bool = True) -> tuple:
    """(estimated microseconds, K ranges) of the pairs-of-SMs form: the number of K ranges per tile (1 = persistent
    pairs, no split, in the tiles that the kernel chooses) whose waves of tiles x K steps cost least.  `may_row`: the product may
    have tiles of equal tokens (bfloat16 output, plain or gated; not the squared relu, nor the q/k/v product with its epilogue)."""
    nkb, tiles = -(-K // 64), -(-M // 256) * -(-N // 256)
    best = (ops.gemm_tcgen05_pair_us(M, N, K, may_row), 1)
    for splits in range(2, ops.PAIR_MAX_SPLITS + 1):
        capacity = ops.gemm_tcgen05_pair_capacity(splits)
        if capacity <= 0 or splits > nkb or tiles > 65535:
            continue
        cost = (-(-tiles * splits // capacity) * (-(-nkb // splits) * _STEP_US["pair"] + _PAIR_SPLIT_WAVE_US)
                + _PAIR_SPLIT_LAUNCH_US)
        if cost < best[0]:
            best = (cost, splits)
    return best


@functools.lru_cache(maxsize=4096)
def tcgen05_form(M: int, N: int, K: int, gated: bool = False, may_row: bool = True) -> str:
    """Which form of the tcgen05 product takes M rows (M > skinny_rows, K a multiple of 8): weights first
    (K split over a cluster; the only form that fills the GPU when M and N give few tiles), or tokens first
    and persistent, on single SMs with 128 x 128 tiles or on pairs of SMs with 256 x 256 tiles or (`may_row`, as above) tiles of
    equal tokens by 256 rows of W.  A small cost model: waves of blocks times K steps."""
    if M <= 128:
        return "weights_first"
    sms = torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
    nkb = -(-K // 64)

    def waves(blocks, slots):
        return -(-blocks // slots)

    cost = {"pair": pair_plan(M, N, K, may_row)[0]}
    if not gated:                                        # the gated epilogue exists for the 256-row tiles
        cost["prompt128"] = waves(-(-M // 128) * -(-N // 128), sms) * nkb * _STEP_US["prompt128"] + _BLOCK_US["prompt128"]
    if M <= 1024:
        splits = ops.gemm_tcgen05_mid_splits(M, N, K)
        blocks = -(-N // 128) * -(-M // 256) * splits
        cost["weights_first"] = waves(blocks, sms) * (-(-nkb // splits) * _STEP_US["weights_first"] + _WEIGHTS_FIRST_US[splits])
    return min(cost, key=cost.get)


@functools.lru_cache(maxsize=4096)
def few_rows_weights_first(M: int, N: int, K: int) -> bool:
    """Whether the weights-first kernel reads W [N, K] sooner than the weight-streaming one even for M <= `skinny_rows` rows, plain or gated.

    The largest matrices from four rows on, up to what three blocks of 128 rows of W an SM hold at once (that / the streaming kernel, us, at 8
    rows: gate and up of the 8B shape, 201 MB, 33.7 / 36.2, of the 14B shape 55.2 / 58.1, its 178 MB down 30.2 / 34.2, 40,960 x 8,192 103 / 111,
    56,832 x 4,096 72.4 / 73.1; one block more, 56,960 x 4,096, 81.8 / 75.0, and 57,344 x 8,192 160 / 154; at 4 rows between 28,672 and 49,152 x
    4,096 the two are within 2 %).  Of one row the largest gained 2 us in one place and lost 2 in another.

    And rows of W that make little more than one wave of the streaming kernel's blocks, three of 16 rows an SM, which it begins anew for a few
    (K 4,096 and 8,192 at 1 row: 7,104 rows of W, one wave, 12.0 / 11.3; 7,168 12.1 / 14.4 and 20.6 / 27.1; 8,192 13.5 / 15.6 and 23.3 / 29.7;
    9,472 14.8 / 16.9 and 26.5 / 31.4; gated 1 us more on both sides).  With K of 2,048 the two are level.  Smaller matrices are slower
    (4,096 x 4,096 8.7 against 7.5, 4,096 x 12,288 18.3 against 17.9)."""
    wave = 3 * torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
    return M >= 4 and 2 * N * K >= 150_000_000 and -(-N // 128) <= wave or K >= 4096 and wave < -(-N // 16) <= wave * 4 // 3


def linear(x: torch.Tensor, w: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
    """out[M, N] = x[M, K] . w[N, K]^T; out is float32 or x's type."""
    if x.dtype == torch.float32:
        if out.dtype != torch.float32:
            raise ops.KernelError("a 32-bit product writes 32-bit output")
        return ops.gemm_f32(x, w, out)
    if x.dtype != torch.bfloat16 or w.dtype != torch.bfloat16:
        raise ops.KernelError(f"linear: unsupported operand types {x.dtype}, {w.dtype}")
    if not x.is_cuda:
        raise ops.KernelError("linear: CUDA tensors only")
    if _bf16_kernel is not None and _bf16_kernel(x, w, out):
        return out
    M, K = x.shape
    if K % 8 != 0:
        return ops.gemm_bf16_any_width(x, w, out)
    if M <= skinny_rows:
        if out.dtype == torch.bfloat16 and few_rows_weights_first(M, w.shape[0], K):
            return ops.gemm_tcgen05_mid(x, w, out)
        return ops.gemm_skinny(x, w, out)
    may_row = out.dtype == torch.bfloat16
    form = tcgen05_form(M, w.shape[0], K, may_row=may_row)
    if form == "weights_first":
        return ops.gemm_tcgen05_mid(x, w, out)
    if form == "pair":
        return ops.gemm_tcgen05_pair(x, w, out, splits=pair_plan(M, w.shape[0], K, may_row)[1])
    return ops.gemm_tcgen05_prompt(x, w, out, tile_n=128)
