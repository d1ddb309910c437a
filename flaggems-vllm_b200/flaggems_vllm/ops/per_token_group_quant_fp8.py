"""FP8 e4m3 quantisation of activations in groups along the last dimension, one fp32 scale per group.

Drop-in for the reference operator of the same module path and name
(src/flaggems_vllm/ops/per_token_group_quant_fp8.py:226-330): same arguments and return values (x_q shaped like x,
scales [..., K / group_size] float32, transposed storage when `column_major_scales`).  bfloat16 inputs and
float8_e4m3fn outputs (the NVIDIA format) only.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from .. import _native

SUPPORTED_FP8_DTYPE = torch.float8_e4m3fn

_call = None  # the native front end, looked up once


def _bind():
    global _call
    _call = _native.host_calls().group_quant
    return _call


def per_token_group_quant_fp8(
    x: torch.Tensor,
    group_size: int,
    eps: float = 1e-10,
    dtype: Optional[torch.dtype] = None,
    column_major_scales: bool = False,
    scale_ue8m0: bool = False,
) -> Tuple[torch.Tensor, torch.Tensor]:
    if dtype is None or dtype == SUPPORTED_FP8_DTYPE:
        result = (_call or _bind())(x, group_size, eps, column_major_scales, scale_ue8m0)
        if result is not None:
            return result
    fp8_dtype = SUPPORTED_FP8_DTYPE if dtype is None else dtype
    assert x.shape[-1] % group_size == 0, (
        f"the last dimension of `x` {x.shape[-1]} must be divisible by `group_size` {group_size}")
    assert x.stride(-1) == 1, "`x` groups must be contiguous"
    assert x.device.type == "cuda", "this operator has no CPU path"
    assert x.dtype == torch.bfloat16 and fp8_dtype == torch.float8_e4m3fn, "bfloat16 -> float8_e4m3fn only"
    assert x.dim() >= 2 and (x.dim() == 2 or x.is_contiguous()), "[M, K] with any row stride, or a contiguous tensor of more dimensions"
    assert not column_major_scales or x.dim() == 2, "column-major scales for [M, K] inputs"
    _native.refuse()


__all__ = ["per_token_group_quant_fp8"]
