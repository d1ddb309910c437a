"""The epilogue quantiser where the number of heads per warp changes, with ragged head counts and both access widths,
against the C oracle."""
from __future__ import annotations

import pytest
import torch

import flaggems_vllm as fg
from flaggems_vllm.testing import workloads
from oracle import c_oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("tokens,groups,per_group", [(1, 1, 1), (3, 3, 1), (5, 8, 16), (127, 8, 16), (131, 8, 16), (300, 5, 11), (700, 8, 16)])
@pytest.mark.parametrize("offset", [0, 8])  # 32-byte and 16-byte aligned rows
def test_tasks(tokens, groups, per_group, offset, packed):
    heads = groups * per_group
    g = torch.Generator(device=DEV).manual_seed(tokens)
    store = torch.randn(tokens * heads * 512 + 16, generator=g, device=DEV).bfloat16()
    o = store[offset : offset + tokens * heads * 512].view(tokens, heads, 512)
    pos = torch.randint(0, 512, (tokens,), generator=g, device=DEV)
    cs = workloads.cos_sin_table(512)
    q, s = fg.fused_inv_rope_fp8_quant(o, pos, cs.to(DEV), groups, per_group, tma_aligned_scales=packed)
    want_q, want_s = c_oracle.inv_rope_fp8_quant(o.cpu(), pos.cpu(), cs, groups, per_group, packed=packed)
    assert torch.equal(q.cpu().view(torch.uint8), want_q)
    assert torch.equal(s.cpu().contiguous().view(torch.int32), want_s.contiguous().view(torch.int32))
