"""Top-k positions inside a request -> slots of the paged cache, and per-token counts.

Drop-in for the reference operator of the same module path and name
(src/flaggems_vllm/ops/deepseek_v4_attention_compute_global_topk_indices_and_lens.py:128-161): same arguments
and return values (int32 indices shaped like `topk_indices`, int32 lens).
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from .. import _native

_call = None  # the native front end, looked up once


def _bind():
    global _call
    _call = _native.host_calls().global_topk
    return _call


def compute_global_topk_indices_and_lens(
    topk_indices: torch.Tensor,
    token_to_req_indices: torch.Tensor,
    block_table: torch.Tensor,
    block_size: int,
    is_valid_token: Optional[torch.Tensor] = None,
) -> Tuple[torch.Tensor, torch.Tensor]:
    result = (_call or _bind())(topk_indices, token_to_req_indices, block_table, block_size, is_valid_token)
    if result is not None:
        return result
    assert topk_indices.ndim == 2
    dev = topk_indices.device
    assert dev.type == "cuda", "this operator has no CPU path"
    assert topk_indices.dtype == torch.int32 and topk_indices.stride(1) == 1, "int32 indices with unit inner stride"
    assert token_to_req_indices.dtype == torch.int32 and token_to_req_indices.is_contiguous()
    assert block_table.dtype == torch.int32 and block_table.dim() == 2 and block_table.stride(1) == 1
    num_tokens = topk_indices.shape[0]
    assert token_to_req_indices.shape == (num_tokens,)
    if is_valid_token is not None:
        assert is_valid_token.dtype == torch.int32 and is_valid_token.shape == (num_tokens,) and is_valid_token.is_contiguous()
    for t in (token_to_req_indices, block_table) + (() if is_valid_token is None else (is_valid_token,)):
        assert t.device == dev, "all tensors must be on the same device"
    assert int(block_size) > 0
    _native.refuse()


__all__ = ["compute_global_topk_indices_and_lens"]
