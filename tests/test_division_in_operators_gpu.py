"""The division shortcut as the operators run it: every bf16 group maximum against every bf16 value up to it, of either sign, through
the public calls, against torch's IEEE division; and that the on-device check of the shortcut runs the operators' own function."""
from __future__ import annotations

import pytest
import torch

import flaggems_vllm as fg
from flaggems_vllm import build

DEV = "cuda:0"


def test_the_check_runs_the_operators_function():
    probe, common = ((build.CSRC / name).read_text() for name in ("division_probe.cu", "dsv4_common.cuh"))
    quant8_by = common[common.index("uint2 quant8_by("):]
    assert "quotients<kDivideFast, TWO_TERM>(" in probe and "quotients<MODE, TWO_TERM>(" in quant8_by[:quant8_by.index("\n}\n")]


def groups_of(first, last):
    """[maxima, groups, 128] bf16: of each maximum every value up to it, the largest again behind them, every second value negative."""
    amax = torch.arange(first, last, device=DEV, dtype=torch.int32)
    values = torch.arange(((last - 1) // 127 + 1) * 127, device=DEV, dtype=torch.int32).view(1, -1, 127)
    values = torch.minimum(values, amax[:, None, None])
    bits = torch.cat((values, amax[:, None, None].expand(-1, values.shape[1], 1)), dim=2)
    odd = torch.arange(128, device=DEV, dtype=torch.int32) + torch.arange(bits.shape[1], device=DEV, dtype=torch.int32)[:, None]
    return torch.where((odd % 2 == 1) & (bits > 0), bits - 0x8000, bits).to(torch.int16).view(torch.bfloat16)


@pytest.mark.gpu
@pytest.mark.parametrize("op", ["group", "epilogue"])
def test_every_group_maximum_and_value(op):
    identity = torch.cat((torch.ones(1, 32, device=DEV), torch.zeros(1, 32, device=DEV)), dim=1)
    for first in range(0, 0x7F80, 480):  # 68 runs of 480 maxima
        x = groups_of(first, first + 480).reshape(-1, 512)
        if op == "group":
            got, scales = fg.per_token_group_quant_fp8(x, 128)
        else:
            got, scales = fg.fused_inv_rope_fp8_quant(x.view(-1, 1, 512), torch.zeros(x.shape[0], dtype=torch.int64, device=DEV), identity, 1, 1, tma_aligned_scales=False)
        want = (x.view(-1, 128).float() / scales.reshape(-1, 1)).to(torch.float8_e4m3fn)
        assert torch.equal(got.reshape(-1, 128).view(torch.uint8), want.view(torch.uint8))
