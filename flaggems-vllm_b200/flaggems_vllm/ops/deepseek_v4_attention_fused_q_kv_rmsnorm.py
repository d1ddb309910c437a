"""Weighted RMSNorm of the q low-rank activations and of the latent KV in one launch.

Drop-in for the reference operator of the same module path and name
(src/flaggems_vllm/ops/deepseek_v4_attention_fused_q_kv_rmsnorm.py:65-103): same arguments,
assertions and return value.  Rows and weights may be bfloat16, float16 or float32, each tensor its own, as the
reference kernel allows; all-bfloat16 (what the DeepSeek-V4 attention layer passes) takes the vectorised kernel.
"""
from __future__ import annotations

from typing import Tuple

import torch

from .. import _native

_DTYPES = (torch.bfloat16, torch.float16, torch.float32)

_call = None  # the native front end, looked up once


def _bind():
    global _call
    _call = _native.host_calls().q_kv_rmsnorm
    return _call


def fused_q_kv_rmsnorm(qr: torch.Tensor, kv: torch.Tensor, q_weight: torch.Tensor, kv_weight: torch.Tensor,
                       eps: float) -> Tuple[torch.Tensor, torch.Tensor]:
    """(qr_out, kv_out) with out = (x * rsqrt(mean(x^2, -1) + eps)) * weight in fp32, rounded to the row's dtype."""
    result = (_call or _bind())(qr, kv, q_weight, kv_weight, eps)
    if result is not None:
        return result
    assert qr.ndim == 2 and kv.ndim == 2
    assert qr.shape[0] == kv.shape[0]
    assert qr.stride(-1) == 1 and kv.stride(-1) == 1
    assert q_weight.is_contiguous() and kv_weight.is_contiguous()
    assert qr.device.type == "cuda", "this operator has no CPU path"
    for t in (qr, kv, q_weight, kv_weight):
        assert t.dtype in _DTYPES, "bfloat16, float16 or float32"
        assert t.device == qr.device, "all tensors must be on the same device"
    assert q_weight.shape == (qr.shape[1],) and kv_weight.shape == (kv.shape[1],)
    _native.refuse()


__all__ = ["fused_q_kv_rmsnorm"]
