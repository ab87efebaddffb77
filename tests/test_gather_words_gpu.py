"""Gathers of one-word rows: every width in one call, more columns than a
register file of them, row counts around a block's share, sources on both sides
of the size that is gathered together, null rows and indexes outside."""
import pytest
import torch

from pageflow_b200 import gather

pytestmark = pytest.mark.gpu
TYPES = (torch.int64, torch.int32, torch.int16, torch.int8, torch.float64)


def _columns(n_src, count):
    g = torch.Generator(device="cuda").manual_seed(n_src)
    cols = []
    for c in range(count):
        t = TYPES[c % len(TYPES)]
        x = torch.randint(-100, 100, (n_src,), device="cuda", generator=g)
        cols.append(x.to(t))
    cols.append(torch.randint(-9, 9, (n_src, 2), device="cuda", generator=g))  # 16 bytes a row
    return cols


@pytest.mark.parametrize("n", [1, 255, 1023, 1024, 1025, 70_003])
@pytest.mark.parametrize("n_src,count", [(1, 1), (999, 4), (50_000, 7)])
def test_widths_and_sizes(n, n_src, count):
    cols = _columns(n_src, count)
    idx = torch.randint(0, n_src, (n,), device="cuda")
    for got, col in zip(gather.index_select_many(cols, idx), cols):
        assert torch.equal(got, col[idx])


@pytest.mark.parametrize("n_src", [3_300_000, 3_600_000])  # 79 and 86 MB of 24 bytes a row
def test_together_and_apart(n_src):
    cols = _columns(n_src, 1)
    idx = torch.randint(0, n_src, (100_001,), device="cuda")
    for got, col in zip(gather.index_select_many(cols, idx), cols):
        assert torch.equal(got, col[idx])


@pytest.mark.parametrize("n_src", [5_000, 5_600_000])
def test_indexes_outside_give_null_rows_and_are_refused(n_src):
    cols = _columns(n_src, 1)
    idx = torch.randint(0, n_src, (5_001,), device="cuda")
    idx[7], idx[1030] = n_src, -5
    out = gather.index_select_many(cols, idx)
    ok = (idx >= 0) & (idx < n_src)
    for got, col in zip(out, cols):
        assert torch.equal(got[ok], col[idx[ok]])
        assert bool((got[~ok] == got[7]).all())
    with pytest.raises(IndexError, match="2 indexes"):
        gather.index_select_many(cols, idx, check_range=True)
    nulls = idx.clone()
    nulls[7], nulls[1030] = gather.NULL, gather.NULL
    with_null = gather.index_with_null_many(cols, nulls)
    for a, b in zip(with_null, out):
        assert torch.equal(a, b)
