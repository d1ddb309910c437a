"""The selection kernels at the widths, row counts and lengths where one hands over to the next, and on rows that mislead
the sample: selected values against torch.topk, positions distinct and inside the row."""
from __future__ import annotations

import pytest
import torch

import flaggems_vllm as fg

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def check(logits, starts, ends, k):
    rows, width = logits.shape
    out = torch.full((rows, k), -7, dtype=torch.int32, device=DEV)
    fg.top_k_per_row_prefill(logits, starts, ends, out, rows, logits.stride(0), logits.stride(1), k)
    got = out.cpu()
    for r in range(rows):
        a, b = int(starts[r]), int(ends[r])
        n = min(k, b - a)
        assert bool((got[r, n:] == -1).all())
        chosen = got[r, :n].long()
        assert chosen.unique().numel() == n and (n == 0 or (int(chosen.min()) >= 0 and int(chosen.max()) < b - a))
        row = logits[r, a:b].cpu()
        assert torch.equal(row[chosen].sort().values, row.topk(n).values.sort().values), (r, a, b)


@pytest.mark.parametrize("rows", [3, 320])  # few rows: wide CTAs and clusters; many: small ones
@pytest.mark.parametrize("width", [2048, 2049, 4096, 4100, 8192, 8196, 16384, 16388, 33000])
def test_widths_where_the_kernel_changes(rows, width):
    g = torch.Generator(device=DEV).manual_seed(width + rows)
    logits = torch.randn(rows, width, generator=g, device=DEV)
    starts = torch.randint(0, 9, (rows,), generator=g, device=DEV, dtype=torch.int32)
    lengths = torch.randint(400, width - 16, (rows,), generator=g, device=DEV, dtype=torch.int32)
    lengths[0], lengths[1], lengths[2] = 512, 513, width - 16
    check(logits, starts, starts + lengths, 512)


@pytest.mark.parametrize("k", [1, 64, 2048, 3839, 3841, 6000])
def test_numbers_selected(k):
    logits = torch.randn(5, 20000, generator=torch.Generator(device=DEV).manual_seed(k), device=DEV)
    ends = torch.tensor([20000, 6001, 19999, 8191, 3], dtype=torch.int32, device=DEV)
    check(logits, torch.zeros(5, dtype=torch.int32, device=DEV), ends, k)


@pytest.mark.parametrize("width", [3000, 8000, 15000, 70000])
def test_rows_that_mislead_the_sample(width):
    g = torch.Generator(device=DEV).manual_seed(7)
    x = torch.randn(8, width, generator=g, device=DEV)
    x[0, 1000:1700] += 8.0  # all of the top k in one run
    x[1] = x[1].sort().values
    x[2] = x[2].sort(descending=True).values
    x[3] = (x[3] * 4).round() / 4  # few distinct values
    x[4, 600:] = -float("inf")  # masked
    x[5, ::4] += 6.0  # what a sample of every fourth value sees
    x[6] = -x[6].abs() * 1e-30
    x[7, 5::2] = float("inf")
    ends = torch.full((8,), width, dtype=torch.int32, device=DEV)
    check(x, torch.zeros_like(ends), ends, 512)


@pytest.mark.parametrize("rows,width", [(300, 8000), (300, 33000), (300, 70001), (450, 140000)])
@pytest.mark.parametrize("length", [8, 128])
def test_values_that_vary_smoothly_along_the_row(rows, width, length):
    """Moving sums over `length` values: neighbours are alike, so the sample, which is taken in runs of neighbours, says less than
    its size and misjudges up to a third of the rows, towards too few candidates as towards too many.  Every row against its
    top k, with as many rows as take small CTAs, wide ones, and two batches in flight."""
    g = torch.Generator(device=DEV).manual_seed(width + length)
    steps = torch.randn(rows, width + length, generator=g, device=DEV).cumsum(dim=1, dtype=torch.float64)
    x = ((steps[:, length:] - steps[:, :-length]) * length**-0.5).float()
    for k in (512, 2048):
        out = torch.full((rows, k), -7, dtype=torch.int32, device=DEV)
        zeros, ends = torch.zeros(rows, dtype=torch.int32, device=DEV), torch.full((rows,), width, dtype=torch.int32, device=DEV)
        fg.top_k_per_row_prefill(x, zeros, ends, out, rows, x.stride(0), x.stride(1), k)
        chosen = out.long().sort(dim=1).values
        assert bool((chosen[:, 0] >= 0).all()) and bool((chosen[:, -1] < width).all()) and bool((chosen[:, 1:] > chosen[:, :-1]).all())
        assert torch.equal(x.gather(1, chosen).sort(dim=1).values, x.topk(k, dim=1).values.sort(dim=1).values)


@pytest.mark.parametrize("rows", [8, 320])
@pytest.mark.parametrize("width", [1500, 3000, 8000, 15000, 20000, 70000])
def test_nans_rank_by_their_sign(width, rows):
    """A NaN is above +inf, one with its sign bit set below -inf, in every kernel and on every route (a pool full of NaNs
    takes the histogram route): the selected bit patterns are those of the largest integer keys of the rows."""
    g = torch.Generator(device=DEV).manual_seed(width)
    x = torch.randn(rows, width, generator=g, device=DEV)
    bits = x.view(torch.int32)
    up, down = 0x7FC00000, -0x400000  # the quiet NaNs
    scattered = torch.rand(rows, width, generator=g, device=DEV)
    bits[0, 7::211] = up
    bits[1, 7::211] = down
    bits[2, 3::97], bits[2, 5::89] = up, down
    bits[3, ::2] = down
    bits[4, 1::2] = up
    bits[5][scattered[5] > 100.0 / width] = down  # fewer numbers than are selected
    bits[6] = torch.where(scattered[6] < 0.5, up, down)
    bits[7, 11::13] = down + torch.arange(len(bits[7, 11::13]), device=DEV, dtype=torch.int32) % 64
    bits[7, 12::130] = -0x800000  # -inf
    k = 512
    out = torch.full((rows, k), -7, dtype=torch.int32, device=DEV)
    zeros, ends = torch.zeros(rows, dtype=torch.int32, device=DEV), torch.full((rows,), width, dtype=torch.int32, device=DEV)
    fg.top_k_per_row_prefill(x, zeros, ends, out, rows, x.stride(0), x.stride(1), k)
    key = torch.where(bits < 0, -0x80000000 - (bits.long() + 1), bits.long())
    chosen = out.long().sort(dim=1).values
    assert bool((chosen[:, 0] >= 0).all()) and bool((chosen[:, -1] < width).all()) and bool((chosen[:, 1:] > chosen[:, :-1]).all())
    assert torch.equal(key.gather(1, chosen).sort(dim=1).values, key.topk(k, dim=1).values.sort(dim=1).values)


@pytest.mark.parametrize("rows,width", [(900, 33000), (444, 70001), (450, 70001), (450, 140000), (700, 65540), (450, 196608), (600, 196612)])
@pytest.mark.parametrize("k", [512, 2048])
def test_rows_that_fill_the_gpu(rows, width, k):
    """The streaming kernel with batches sent to L2 ahead of their loads: small CTAs, wide ones with one batch in flight (444 rows,
    the most they take) and with two, and these with the longest rows first.  Ranges of every length, most of them starting off a
    16-byte boundary, ties included."""
    g = torch.Generator(device=DEV).manual_seed(rows + width)
    x = torch.randn(rows, width, generator=g, device=DEV)
    x[::3] = (x[::3] * 64).round() / 64
    starts = torch.randint(0, 9, (rows,), generator=g, device=DEV, dtype=torch.int32)
    lengths = torch.randint(k, width - 9, (rows,), generator=g, device=DEV, dtype=torch.int32)
    lengths[:4] = torch.tensor([k, k + 1, width - 9, 4097], dtype=torch.int32, device=DEV)
    out = torch.full((rows, k), -7, dtype=torch.int32, device=DEV)
    fg.top_k_per_row_prefill(x, starts, starts + lengths, out, rows, x.stride(0), x.stride(1), k)
    chosen = out.long().sort(dim=1).values
    assert bool((chosen[:, 0] >= 0).all()) and bool((chosen[:, -1] < lengths).all()) and bool((chosen[:, 1:] > chosen[:, :-1]).all())
    got = x.gather(1, chosen + starts[:, None]).sort(dim=1).values
    for r in range(rows):
        a, n = int(starts[r]), int(lengths[r])
        assert torch.equal(got[r], x[r, a : a + n].topk(k).values.sort().values), (r, a, n)
