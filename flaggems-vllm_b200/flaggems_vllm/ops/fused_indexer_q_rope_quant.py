"""Sparse-indexer prologue: GPT-J RoPE on the index-q tail + FP8 (per head) or MXFP4 (per 32) quantisation.

Drop-in for the reference operator of the same module path and name
(src/flaggems_vllm/ops/fused_indexer_q_rope_quant.py:283-410): same arguments, return structure, dtypes
and weight-fold semantics.  bf16 index_q, head_dim 64 / 128 / 256.
"""
from __future__ import annotations

import torch

from .. import _native

_WEIGHT_DTYPES = (torch.bfloat16, torch.float16, torch.float32)

_call = None  # the native front end, looked up once


def _bind():
    global _call
    _call = _native.host_calls().indexer_q_rope_quant
    return _call


def fused_indexer_q_rope_quant(
    positions: torch.Tensor,
    index_q: torch.Tensor,
    index_q_cos_sin_cache: torch.Tensor,
    index_weights: torch.Tensor,
    index_weights_softmax_scale: float,
    index_weights_head_scale: float,
    use_fp4: bool = False,
):
    """Returns (q_quant, weights_out).

    FP8 (default): q_quant float8_e4m3fn like index_q, one power-of-two scale per (token, head) that is
    folded into weights_out = weights * q_scale * softmax_scale * head_scale.
    MXFP4: q_quant = (uint8 [T, H, D/2] with two e2m1 codes per byte, int32 [T, H] holding the four UE8M0
    block-scale bytes when D = 128, else uint8 [T, H, D/32] viewed as int32); weights_out = weights *
    softmax_scale * head_scale.
    """
    result = (_call or _bind())(positions, index_q, index_q_cos_sin_cache, index_weights, index_weights_softmax_scale,
                                index_weights_head_scale, use_fp4)
    if result is not None:
        return result
    assert positions.ndim == 1
    assert index_q.ndim == 3
    assert index_q_cos_sin_cache.ndim == 2
    num_tokens = positions.shape[0]
    num_heads, head_dim = index_q.shape[1], index_q.shape[2]
    rot_dim = index_q_cos_sin_cache.shape[-1]

    if use_fp4 and not index_q.is_cuda:
        raise RuntimeError("MXFP4 fused_indexer_q_rope_quant requires CUDA")
    assert index_q.device.type == "cuda", "this operator has no CPU path"
    assert index_q.dtype == torch.bfloat16 and index_q.stride(2) == 1 and index_q.shape[0] == num_tokens
    assert positions.dtype == torch.int64 and positions.is_contiguous()
    assert index_q_cos_sin_cache.dtype in (torch.float32, torch.bfloat16) and index_q_cos_sin_cache.stride(1) == 1
    assert index_weights.dtype in _WEIGHT_DTYPES and index_weights.shape == (num_tokens, num_heads)
    assert index_weights.stride(1) == 1
    assert head_dim in (64, 128, 256), "head_dim must be 64, 128 or 256"
    assert rot_dim % 2 == 0 and rot_dim <= head_dim and (head_dim - rot_dim) % (head_dim // 32) == 0
    for t in (positions, index_q_cos_sin_cache, index_weights):
        assert t.device == index_q.device, "all tensors must be on the same device"
    _native.refuse()


__all__ = ["fused_indexer_q_rope_quant"]
