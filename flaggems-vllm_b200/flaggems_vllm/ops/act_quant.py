"""Block-wise FP8 activation quantisation (DeepSeek's `act_quant`).

Drop-in for the reference operator of the same module path and name
(src/flaggems_vllm/ops/act_quant.py:113-175): same arguments and return values (float8_e4m3fn tensor shaped like x,
float32 scales [..., N / block_size]).  bfloat16 inputs only.  The name keeps the reference's `_triton` suffix because
that is what callers import; nothing here is Triton.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from .. import _native

_call = None  # the native front end, looked up once


def _bind():
    global _call
    _call = _native.host_calls().act_quant
    return _call


def act_quant_triton(x: torch.Tensor, block_size: int = 128, scale_fmt: Optional[str] = None) -> Tuple[torch.Tensor, torch.Tensor]:
    result = (_call or _bind())(x, block_size, scale_fmt is not None)
    if result is not None:
        return result
    assert x.is_contiguous(), "Input tensor must be contiguous"
    assert x.size(-1) % block_size == 0, f"Last dimension size must be divisible by block_size (block_size={block_size})"
    assert x.device.type == "cuda", "this operator has no CPU path"
    assert x.dtype == torch.bfloat16, "bfloat16 only"
    _native.refuse()


__all__ = ["act_quant_triton"]
