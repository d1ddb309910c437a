"""The indexer q prologue where the number of heads per warp changes, with ragged head counts and both load widths, against the C
oracle."""
from __future__ import annotations

import pytest
import torch

import flaggems_vllm as fg
from flaggems_vllm.testing import workloads
from oracle import c_oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("fp4", [False, True])
@pytest.mark.parametrize("tokens,heads", [(1, 1), (3, 9), (5, 64), (895, 64), (897, 64), (1023, 64), (1025, 64), (3075, 64), (3327, 64), (3329, 64), (9217, 64), (12289, 64), (11000, 75)])
@pytest.mark.parametrize("offset", [0, 8])  # rows on 32-byte and on 16-byte boundaries
def test_heads_per_task(tokens, heads, fp4, offset):
    if tokens > 4000 and offset:
        pytest.skip("one width is enough at this size")
    g = torch.Generator(device=DEV).manual_seed(tokens)
    store = torch.randn(tokens * heads * 128 + 16, generator=g, device=DEV).bfloat16()
    q = store[offset : offset + tokens * heads * 128].view(tokens, heads, 128)
    w = torch.randn(tokens, heads, generator=g, device=DEV).bfloat16()
    pos = torch.randint(0, 512, (tokens,), generator=g, device=DEV)
    cs = workloads.cos_sin_table(512)
    got, got_w = fg.fused_indexer_q_rope_quant(pos, q, cs.to(DEV), w, 0.0884, 0.125, use_fp4=fp4)
    want, want_s, want_w = c_oracle.indexer_q_rope_quant(pos.cpu(), q.cpu(), cs, w.cpu(), 0.0884, 0.125, use_fp4=fp4)
    assert torch.equal(got_w.cpu(), want_w)
    if fp4:
        assert torch.equal(got[0].cpu(), want) and torch.equal(got[1].cpu().contiguous().view(torch.uint8).flatten(), want_s.contiguous().view(torch.uint8).flatten())
    else:
        assert torch.equal(got.cpu().view(torch.uint8), want)
