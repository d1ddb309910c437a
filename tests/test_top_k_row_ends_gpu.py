"""Selection where the largest values are the first and the last ones of a row whose ends lie anywhere inside 16 bytes, and where NaNs of
both signs and infinities share a row: on each kernel for rows too long for registers, few and many rows, one CTA or a cluster."""
from __future__ import annotations

import pytest
import torch

import flaggems_vllm as fg

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# rows, width: clusters of CTAs with two batches in flight, CTAs of 256 threads, CTAs of 512 threads in one wave, in more, and in more
# with the longest rows first
SHAPES = [(3, 40003), (320, 17000), (320, 70001), (460, 70001), (460, 140002), (592, 131072)]


def rows_of(rows, width, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.empty(rows, width, device=DEV).normal_(generator=g)
    r = torch.arange(rows, device=DEV)
    starts = (r % 5).to(torch.int32)
    ends = (width - (r // 5) % 7 - (r % 3) * (width // 5)).to(torch.int32)  # lengths differ, remainders of 4 all occur
    return x, starts, ends


@pytest.mark.parametrize("rows,width", SHAPES)
def test_ends_of_rows(rows, width):
    x, starts, ends = rows_of(rows, width, rows + width)
    r, k = torch.arange(rows, device=DEV), 512
    for i in range(3):
        x[r, starts.long() + i] = 50.0 + i
        x[r, ends.long() - 1 - i] = 60.0 + i
    before, behind = starts > 0, ends < width
    x[r[before], starts[before].long() - 1] = 99.0  # outside the range
    x[r[behind], ends[behind].long()] = 99.0
    picked = torch.empty(rows, k, dtype=torch.int32, device=DEV)
    fg.top_k_per_row_prefill(x, starts, ends, picked, rows, x.stride(0), 1, k)
    inside = (r.new_zeros(1) + torch.arange(width, device=DEV)).unsqueeze(0)
    masked = x.masked_fill((inside < starts.unsqueeze(1)) | (inside >= ends.unsqueeze(1)), float("-inf"))
    want = masked.topk(k, dim=1).values
    got = x.gather(1, picked.long() + starts.unsqueeze(1)).sort(dim=1, descending=True).values
    assert torch.equal(got, want)
    assert (picked.sort(dim=1).values.diff(dim=1) > 0).all()


@pytest.mark.parametrize("rows,width", SHAPES)
def test_values_that_are_not_finite(rows, width):
    """400 positive NaNs or infinities a row and 100 negative ones, k 512: all of the former, none of the latter."""
    x, starts, ends = rows_of(rows, width, rows)
    r, k = torch.arange(rows, device=DEV), 512
    nan = torch.tensor([0x7FC00000, 0x7F800000, -0x00400000, -0x00800000], dtype=torch.int32, device=DEV).view(torch.float32)  # nan, inf, -nan, -inf
    place = torch.randperm(int((ends - starts).min()), generator=torch.Generator(device=DEV).manual_seed(3), device=DEV)[:500]
    bits = x.view(torch.int32)
    kind = torch.arange(500, device=DEV) % 2 + 2 * (torch.arange(500, device=DEV) >= 400)
    for j in range(500):
        bits[r, starts.long() + place[j]] = nan.view(torch.int32)[kind[j]]
    picked = torch.empty(rows, k, dtype=torch.int32, device=DEV)
    fg.top_k_per_row_prefill(x, starts, ends, picked, rows, x.stride(0), 1, k)
    flag = torch.zeros(rows, width, dtype=torch.bool, device=DEV)
    flag.scatter_(1, picked.long(), True)
    assert flag[:, place[:400]].all() and not flag[:, place[400:]].any()
    assert (picked.sort(dim=1).values.diff(dim=1) > 0).all()
