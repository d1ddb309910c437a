"""The two access widths of the group quantiser and its two numbers of groups in flight, against the C oracle: row counts
either side of the change, bases and row strides that are multiples of 32 bytes and of 16 bytes only."""
from __future__ import annotations

import pytest
import torch

import flaggems_vllm as fg
from oracle import c_oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("group", [64, 128, 256, 512])
@pytest.mark.parametrize("offset,stride", [(0, 1024), (8, 1024), (0, 1032)])
@pytest.mark.parametrize("rows", [1, 3, 4099])
@pytest.mark.parametrize("ue8m0", [True, False])
def test_access_widths(group, offset, stride, rows, ue8m0):
    cols = 1024
    g = torch.Generator(device=DEV).manual_seed(rows + group)
    store = torch.randn(rows * stride + 16, generator=g, device=DEV).bfloat16()
    x = store[offset : offset + rows * stride].view(rows, stride)[:, :cols] if stride > cols else store[offset : offset + rows * stride].view(rows, cols)
    q, s = fg.per_token_group_quant_fp8(x, group, scale_ue8m0=ue8m0)
    want_q, want_s = c_oracle.per_token_group_quant_fp8(x.cpu().contiguous(), group, scale_ue8m0=ue8m0)
    assert torch.equal(q.cpu().view(torch.uint8), want_q) and torch.equal(s.cpu().view(torch.int32), want_s.view(torch.int32))
