"""Selection from short rows (up to 4096 values): lengths around the pieces a thread takes, every alignment of a row's ends, strided
rows, and rows whose k-th largest value is minus infinity or a NaN with its sign bit set (where values beside the row would count)."""
from __future__ import annotations

import pytest
import torch

import flaggems_vllm as fg

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ranks(x):
    """Integers in the order of the selection: of the floats, and NaNs by their sign above and below all of them."""
    bits = x.contiguous().view(torch.int32).long() & 0xFFFFFFFF
    return torch.where(bits >= 1 << 31, 0xFFFFFFFF - bits, bits + (1 << 31))


def check(x, starts, ends, k):
    rows = x.shape[0]
    picked = torch.empty(rows, k, dtype=torch.int32, device=DEV)
    fg.top_k_per_row_prefill(x, starts, ends, picked, rows, x.stride(0), x.stride(1), k)
    key = ranks(x).cpu()
    for r in range(rows):
        a, b = int(starts[r]), int(ends[r])
        n = min(k, b - a)
        got = picked[r].cpu()
        assert (got[n:] == -1).all()
        got = got[:n].long()
        assert got.unique().numel() == n and (n == 0 or (got.min() >= 0 and got.max() < b - a))
        assert torch.equal(key[r, a:b][got].sort().values, key[r, a:b].sort().values[b - a - n:]), f"row {r}"


@pytest.mark.parametrize("rows", [5, 300])  # CTAs of 512 threads; of 128 or 256
@pytest.mark.parametrize("width", [513, 1027, 2047, 2048, 2049, 4093])
def test_lengths_and_alignments(rows, width):
    g = torch.Generator(device=DEV).manual_seed(width)
    x = torch.empty(rows, width, device=DEV).normal_(generator=g)
    r = torch.arange(rows, device=DEV)
    starts, ends = (r % 4).to(torch.int32), (width - (r * 37) % (width // 2)).to(torch.int32)
    check(x, starts, ends, 512)
    check(x.t().contiguous().t(), starts, ends, 100)  # values of a row not adjacent


@pytest.mark.parametrize("rows", [5, 300])
@pytest.mark.parametrize("finite", [0, 100, 511, 512, 600])
def test_the_lowest_values(rows, finite):
    """`finite` ordinary values a row, the others -inf, some of them -NaN: k 512 reaches down to them where there are fewer."""
    g = torch.Generator(device=DEV).manual_seed(finite)
    width = 2051
    x = torch.full((rows, width), float("-inf"), device=DEV)
    place = torch.randperm(width, generator=g, device=DEV)
    x[:, place[:finite]] = torch.empty(rows, finite, device=DEV).normal_(generator=g)
    x.view(torch.int32)[:, place[finite : finite + 700]] = -1
    r = torch.arange(rows, device=DEV)
    check(x, (r % 4).to(torch.int32), (width - r % 4).to(torch.int32), 512)
