"""The indexer q prologue on both sides of the sizes at which a warp's number of heads changes, against the C oracle, and its
packed arithmetic on subnormal, infinite and NaN values, against the kernel that works value by value."""
from __future__ import annotations

import pytest
import torch

import flaggems_vllm as fg
from flaggems_vllm.testing import workloads
from oracle import c_oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _bytes(got, fp4):
    return [x.cpu().contiguous().view(torch.uint8).flatten() for x in (got[0] if fp4 else (got[0],))] + [got[1].cpu()]


@pytest.mark.parametrize("fp4", [False, True])
@pytest.mark.parametrize("tokens,heads", [(223, 64), (224, 64), (1381, 64), (1382, 64), (1776, 64), (1777, 64), (2763, 64), (3552, 64), (3553, 64), (2500, 75), (1500, 50)])
def test_both_sides_of_the_lines(tokens, heads, fp4):
    g = torch.Generator(device=DEV).manual_seed(tokens)
    q = torch.randn(tokens, heads, 128, generator=g, device=DEV).bfloat16()
    w = torch.randn(tokens, heads, generator=g, device=DEV).bfloat16()
    pos = torch.randint(0, 512, (tokens,), generator=g, device=DEV)
    cs = workloads.cos_sin_table(512)
    got = _bytes(fg.fused_indexer_q_rope_quant(pos, q, cs.to(DEV), w, 0.0884, 0.125, use_fp4=fp4), fp4)
    want, want_s, want_w = c_oracle.indexer_q_rope_quant(pos.cpu(), q.cpu(), cs, w.cpu(), 0.0884, 0.125, use_fp4=fp4)
    assert torch.equal(got[0], want.contiguous().view(torch.uint8).flatten()) and torch.equal(got[-1], want_w)
    if fp4:
        assert torch.equal(got[1], want_s.contiguous().view(torch.uint8).flatten())


@pytest.mark.parametrize("fp4", [False, True])
@pytest.mark.parametrize("tokens,heads", [(1979, 96), (2533, 75), (1125, 80), (1382, 48), (1875, 48), (2763, 48), (4737, 48), (12289, 48), (5520, 40), (2763, 24), (4737, 24), (14336, 1), (3001, 3)])
def test_other_numbers_of_heads(tokens, heads, fp4):
    """Numbers of heads that leave a short last task, one task a token, and tasks of 40 and 48 heads, with and without requests to L2."""
    test_both_sides_of_the_lines(tokens, heads, fp4)


@pytest.mark.parametrize("fp4", [False, True])
@pytest.mark.parametrize("offset", [0, 8])
@pytest.mark.parametrize("tokens,heads", [(914, 64), (915, 64), (1036, 64), (1037, 64), (1830, 64), (2072, 64), (3661, 64), (4144, 64), (4000, 16), (1980, 24), (1000, 50)])
def test_one_or_two_waves_of_seven_ctas(tokens, heads, offset, fp4):
    """Either side of the sizes that take seven CTAs per SM, on both row alignments."""
    g = torch.Generator(device=DEV).manual_seed(tokens + offset)
    store = torch.empty(tokens * heads * 128 + offset, device=DEV, dtype=torch.bfloat16).normal_(generator=g)
    q = store[offset:].view(tokens, heads, 128)
    w = torch.randn(tokens, heads, generator=g, device=DEV)
    pos = torch.randint(0, 512, (tokens,), generator=g, device=DEV)
    cs = workloads.cos_sin_table(512)
    got = _bytes(fg.fused_indexer_q_rope_quant(pos, q, cs.to(DEV), w, 0.0884, 0.125, use_fp4=fp4), fp4)
    want, want_s, want_w = c_oracle.indexer_q_rope_quant(pos.cpu(), q.cpu(), cs, w.cpu(), 0.0884, 0.125, use_fp4=fp4)
    assert torch.equal(got[0], want.contiguous().view(torch.uint8).flatten()) and torch.equal(got[-1], want_w)
    if fp4:
        assert torch.equal(got[1], want_s.contiguous().view(torch.uint8).flatten())


@pytest.mark.parametrize("fp4", [False, True])
def test_special_values(fp4):
    tokens, heads = 96, 64
    g = torch.Generator(device=DEV).manual_seed(7)
    bits = torch.randint(-32768, 32768, (tokens, heads, 128), generator=g, device=DEV, dtype=torch.int32).to(torch.int16)
    bits[0::4] &= -32513  # subnormals and zeros of either sign: no exponent bits above the lowest one (0x80ff)
    bits[1::4] |= 0x7F80  # infinities and NaNs
    bits[2::4, :, 5] = 0x7FC0  # one NaN among finite values of every magnitude
    q = bits.view(torch.bfloat16)
    store = torch.empty(tokens * heads * 128 + 4, device=DEV, dtype=torch.bfloat16)
    other = store[4:].view(tokens, heads, 128).copy_(q)  # on an 8-byte boundary: one warp per row, value by value
    w = torch.randn(tokens, heads, generator=g, device=DEV)
    pos = torch.randint(0, 512, (tokens,), generator=g, device=DEV)
    cs = workloads.cos_sin_table(512).to(DEV)
    got, want = (_bytes(fg.fused_indexer_q_rope_quant(pos, x, cs, w, 0.0884, 0.125, use_fp4=fp4), fp4) for x in (q, other))
    assert torch.equal(other.view(torch.int16), bits)
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
