"""Rows [compressed top-k entries | sliding-window entries | -1 padding] of indices into the gathered key buffer.

Drop-in for the reference operator of the same module path and name
(src/flaggems_vllm/ops/deepseek_v4_attention_combine_topk_swa_indices.py:109-161): same arguments and return
values (int32 [num_tokens, round_up(topk + window_size, 128)] and int32 lens).  Rows of tokens that no request
covers are left uninitialised, as in the reference.
"""
from __future__ import annotations

from typing import Tuple

import torch

from .. import _native

_call = None  # the native front end, looked up once


def _bind():
    global _call
    _call = _native.host_calls().combine_topk_swa
    return _call


def combine_topk_swa_indices(
    topk_indices: torch.Tensor,
    query_start_loc: torch.Tensor,
    seq_lens: torch.Tensor,
    gather_lens: torch.Tensor,
    window_size: int,
    compress_ratio: int,
    topk: int,
    M: int,
    N: int,
) -> Tuple[torch.Tensor, torch.Tensor]:
    result = (_call or _bind())(topk_indices, query_start_loc, seq_lens, gather_lens, window_size, compress_ratio, topk, M, N)
    if result is not None:
        return result
    assert topk_indices.ndim == 2
    dev = topk_indices.device
    assert dev.type == "cuda", "this operator has no CPU path"
    num_reqs = seq_lens.shape[0]
    assert topk_indices.dtype == torch.int32 and topk_indices.stride(1) == 1, "int32 indices with unit inner stride"
    assert topk <= topk_indices.shape[1], "topk entries are read from every row"
    assert topk + window_size >= 0, "a row of the result holds topk + window_size entries"
    for t in (query_start_loc, seq_lens, gather_lens):
        assert t.dtype == torch.int32 and t.dim() == 1 and t.is_contiguous() and t.device == dev
    assert query_start_loc.shape[0] >= num_reqs + 1 and gather_lens.shape[0] >= num_reqs
    _native.refuse()


__all__ = ["combine_topk_swa_indices"]
