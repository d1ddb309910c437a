"""The weighted norms at the row sizes and alignments where the kernel changes, either side of the token count that decides
when the weights are fetched, against the C oracle."""
from __future__ import annotations

import pytest
import torch

import flaggems_vllm as fg
from flaggems_vllm.testing import compare
from oracle import c_oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("q_size,kv_size", [(16, 512), (512, 512), (528, 16), (1024, 500), (1000, 504), (8, 1544), (1536, 512), (1552, 512), (2048, 1536), (2064, 512)])
@pytest.mark.parametrize("offset", [0, 8])  # rows on 32-byte and on 16-byte boundaries
@pytest.mark.parametrize("tokens", [1, 5, 4099])
def test_row_sizes(q_size, kv_size, offset, tokens):
    g = torch.Generator(device=DEV).manual_seed(q_size + tokens)
    stride = q_size + kv_size + 16 - (q_size + kv_size) % 16 + offset
    x = torch.randn(tokens, stride, generator=g, device=DEV).bfloat16()
    q, kv = x[:, :q_size], x[:, stride - kv_size :]
    wq, wk = torch.randn(q_size, generator=g, device=DEV).bfloat16(), torch.randn(kv_size, generator=g, device=DEV).bfloat16()
    for got, rows, w in zip(fg.fused_q_kv_rmsnorm(q, kv, wq, wk, 1e-6), (q, kv), (wq, wk)):
        want = c_oracle.weighted_rmsnorm(rows.cpu().contiguous(), w.cpu(), 1e-6)
        assert int(compare.bf16_ulp_distance(got.cpu(), want).max()) <= 1


@pytest.mark.parametrize("tokens", [1480, 1481, 2072, 2073, 4096, 4097])
def test_both_sides_of_the_lines(tokens):
    """Rows of 1536 and 512 either side of the launch sizes that decide when the weights are fetched."""
    g = torch.Generator(device=DEV).manual_seed(tokens)
    q, kv = torch.randn(tokens, 1536, generator=g, device=DEV).bfloat16(), torch.randn(tokens, 512, generator=g, device=DEV).bfloat16()
    wq, wk = torch.randn(1536, generator=g, device=DEV).bfloat16(), torch.randn(512, generator=g, device=DEV).bfloat16()
    for got, rows, w in zip(fg.fused_q_kv_rmsnorm(q, kv, wq, wk, 1e-6), (q, kv), (wq, wk)):
        assert int(compare.bf16_ulp_distance(got.cpu(), c_oracle.weighted_rmsnorm(rows.cpu(), w.cpu(), 1e-6)).max()) <= 1


@pytest.mark.parametrize("q_size,tokens", [(1536, 740), (1536, 741), (1536, 1184), (1536, 1185), (512, 2961), (512, 4097), (1024, 2073), (1024, 2961), (2048, 1185), (2048, 1777)])
def test_lines_of_the_other_forms(q_size, tokens):
    """Either side of the sizes that decide how many CTAs an SM holds with rows of 1536, and where a wave of the other widths ends."""
    g = torch.Generator(device=DEV).manual_seed(tokens)
    q, kv = torch.randn(tokens, q_size, generator=g, device=DEV).bfloat16(), torch.randn(tokens, 512, generator=g, device=DEV).bfloat16()
    wq, wk = torch.randn(q_size, generator=g, device=DEV).bfloat16(), torch.randn(512, generator=g, device=DEV).bfloat16()
    for got, rows, w in zip(fg.fused_q_kv_rmsnorm(q, kv, wq, wk, 1e-6), (q, kv), (wq, wk)):
        assert int(compare.bf16_ulp_distance(got.cpu(), c_oracle.weighted_rmsnorm(rows.cpu(), w.cpu(), 1e-6)).max()) <= 1
