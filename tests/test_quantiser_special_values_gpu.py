"""The group and epilogue quantisers on infinities, NaNs, zeros of either sign and the ends of the bf16 range, on every kernel form,
against the C oracle: of a group with an infinity the finite values are x / inf = 0, the infinities NaN."""
from __future__ import annotations

import pytest
import torch

import flaggems_vllm as fg
from flaggems_vllm.testing import workloads
from oracle import c_oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def special_rows(rows, cols):
    g = torch.Generator().manual_seed(cols)
    x = torch.randn(rows, cols, generator=g).bfloat16()
    bits = torch.randint(-32768, 32768, (rows, cols), generator=g, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    x[1::8, 5::97] = float("inf")
    x[2::8, 3::64] = -float("inf")
    x[3::8] = bits[3::8]  # any bf16 value, infinities and NaNs among them
    x[4::8, ::7] = float("nan")
    x[5::8] = x[5::8].clone() * 2.0**126 * torch.rand(x[5::8].shape, generator=g).bfloat16()
    x[6::8] = x[6::8].clone() * 2.0**-126
    x[7::8, ::2] = -0.0
    x[7::16] = float("inf")
    return x


def same(got, want, fp32_scales):
    """Equal bytes, NaNs of either sign taken as one; with fp32 scales a zero's sign is not compared, since the division's last step is a sum
    that makes +0 of -0."""
    def canonical(b):
        b = b.cpu().contiguous().view(torch.uint8).flatten().clone()
        b[(b & 0x7F) == 0x7F] = 0x7F
        if fp32_scales:
            b[b == 0x80] = 0
        return b

    return torch.equal(canonical(got), canonical(want))


@pytest.mark.parametrize("ue8m0", [False, True])
@pytest.mark.parametrize("group,offset", [(64, 0), (128, 0), (256, 0), (512, 0), (128, 8), (128, 1), (48, 0)])
def test_group_quantiser(group, offset, ue8m0):
    cols = 3 * 768 if group == 48 else 1024
    x = torch.empty(131 * cols + offset, dtype=torch.bfloat16)[offset:].view(131, cols).copy_(special_rows(131, cols))
    on_device = torch.empty(131 * cols + offset, dtype=torch.bfloat16, device=DEV)[offset:].view(131, cols).copy_(x)
    got, scales = fg.per_token_group_quant_fp8(on_device, group, scale_ue8m0=ue8m0)
    want, want_scales = c_oracle.per_token_group_quant_fp8(x, group, scale_ue8m0=ue8m0)
    assert torch.equal(scales.cpu(), want_scales) and same(got, want, not ue8m0)
    got, scales = fg.act_quant_triton(on_device, group, "ue8m0" if ue8m0 else None)
    want, want_scales = c_oracle.act_quant(x, group, "ue8m0" if ue8m0 else None)
    assert torch.equal(scales.cpu(), want_scales) and same(got, want, False)


@pytest.mark.parametrize("eps", [1e-10, 1e-4])
@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("offset", [0, 8, 1])
def test_epilogue(offset, packed, eps):
    tokens, heads = 67, 6
    o = special_rows(tokens * heads, 512)
    on_device = torch.empty(o.numel() + offset, dtype=torch.bfloat16, device=DEV)[offset:].view(tokens, heads, 512).copy_(o.view(tokens, heads, 512))
    pos = torch.arange(tokens)
    cs = workloads.cos_sin_table(128)
    got, scales = fg.fused_inv_rope_fp8_quant(on_device, pos.to(DEV), cs.to(DEV), 2, 3, eps=eps, tma_aligned_scales=packed)
    want, want_scales = c_oracle.inv_rope_fp8_quant(o.view(tokens, heads, 512), pos, cs, 2, 3, eps=eps, packed=packed)
    assert torch.equal(scales.cpu().contiguous(), want_scales) and same(got, want, not packed)
