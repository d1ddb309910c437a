"""The cache readers and index operators where their access width or their way to find a request changes, against the C
oracle."""
from __future__ import annotations

import pytest
import torch

import flaggems_vllm as fg
from oracle import c_oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("batch", [1, 31, 32, 33, 255, 256])
@pytest.mark.parametrize("longest,extra", [(3, 0), (70, 5)])
def test_indexer_gather_requests(batch, longest, extra):
    g = torch.Generator().manual_seed(batch + longest)
    lens = torch.randint(0, longest + 1, (batch,), generator=g)  # empty requests among them
    cu = torch.cat([torch.zeros(1), lens.cumsum(0)]).to(torch.int32)
    table = torch.randint(-1, 40, (batch, 8), generator=g).to(torch.int32)  # -1: an unused entry, left alone
    cache = torch.randint(0, 256, (40, 16, 132), generator=g, dtype=torch.uint8)
    tokens = int(cu[-1]) + extra
    k, s = torch.full((tokens, 128), 7, dtype=torch.uint8), torch.full((tokens, 4), 9, dtype=torch.uint8)
    gk, gs = k.to(DEV), s.to(DEV)
    fg.cp_gather_indexer_k_quant_cache(cache.to(DEV), gk, gs, table.to(DEV), cu.to(DEV))
    for t in range(int(cu[-1])):
        b = int((cu <= t).sum()) - 1
        off = t - int(cu[b])
        block = int(table[b, off // 16])
        if block >= 0:
            flat = cache[block].flatten()
            k[t], s[t] = flat[off % 16 * 128 : off % 16 * 128 + 128], flat[2048 + off % 16 * 4 : 2048 + off % 16 * 4 + 4]
    assert torch.equal(gk.cpu(), k) and torch.equal(gs.cpu(), s)


@pytest.mark.parametrize("tokens,longest", [(1, 1), (15, 16), (17, 200)])
@pytest.mark.parametrize("pad", [0, 8])  # output rows on 32-byte and on 16-byte boundaries
def test_dequantize_access_width(tokens, longest, pad):
    g = torch.Generator().manual_seed(tokens)
    cache = torch.randint(0, 256, (16, 64 * 584), generator=g, dtype=torch.uint8) & 0xBF
    table = torch.randperm(16, generator=g)[:8].view(2, 4).to(torch.int32)
    lens = torch.tensor([tokens, longest], dtype=torch.int32)
    out = torch.zeros(2, longest + 3, 512 + pad, dtype=torch.bfloat16)
    got = out.to(DEV)
    fg.dequantize_and_gather_k_cache(got[..., :512], cache.to(DEV), lens.to(DEV), None, table.to(DEV), 64, offset=2)
    want = out[..., :512].contiguous()
    c_oracle.dequantize_and_gather(want, cache, lens, None, table, 64, offset=2)
    assert torch.equal(got[..., :512].cpu().view(torch.int16), want.view(torch.int16)) and not bool(got[..., 512:].any())


@pytest.mark.parametrize("topk", [8, 12, 520, 768, 777, 2048])
@pytest.mark.parametrize("requests", [1, 254, 256])
def test_index_rows(topk, requests):
    g = torch.Generator().manual_seed(topk + requests)
    tokens = requests + 9
    local = torch.randint(-1, 2048, (tokens, topk), generator=g).to(torch.int32)
    request = torch.randint(0, requests, (tokens,), generator=g).to(torch.int32)
    table = torch.randint(0, 500, (requests, 32), generator=g).to(torch.int32)
    out, lens = fg.compute_global_topk_indices_and_lens(local.to(DEV), request.to(DEV), table.to(DEV), 64)
    want, want_lens = c_oracle.compute_global_topk_indices_and_lens(local, request, table, 64)
    assert torch.equal(out.cpu(), want) and torch.equal(lens.cpu(), want_lens)
    start = torch.cat([torch.zeros(1), torch.full((requests,), 1.0).index_add(0, torch.tensor([requests - 1]), torch.tensor([9.0])).cumsum(0)]).to(torch.int32)
    seq = torch.randint(1, 5000, (requests,), generator=g).to(torch.int32) + 10
    gather = torch.minimum(seq, torch.full_like(seq, 137))
    args = (128, 4, topk, 9000, 1300)
    rows, n = fg.combine_topk_swa_indices(local.to(DEV), start.to(DEV), seq.to(DEV), gather.to(DEV), *args)
    want, want_n = c_oracle.combine_topk_swa_indices(local, start, seq, gather, *args)
    assert torch.equal(rows.cpu(), want) and torch.equal(n.cpu(), want_n)
