"""Paged scans of pages cut into four to eight parts, the last of them empty or
ragged, in whole and in the last row group, against the oracle; a bad page is
counted four times whatever the parts."""
import pytest
import torch

import oracle
from pageflow_b200 import paged
from tests.test_paged_gpu import _check, _edge_columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rpp", [16384, 2 * 16384, 3 * 16384, 5 * 16384, 131072])
@pytest.mark.parametrize("tail", [0, 1, 4097, 20_000])
def test_parts(rpp, tail):
    n = 2 * rpp + tail
    cols = _edge_columns(n)
    t = paged.PagedTable.from_columns(cols, rows_per_page=rpp)
    lo, hi = n // 7 // 700, 5 * (n // 7) // 700
    parts = paged.paged_scan(t, "filter", lo, hi, "key", B=16, groups_per_batch=2)
    torch.cuda.synchronize()
    want = oracle.paged_scan(cols, n, rpp, 2, "filter", lo, hi, "key", 16)
    _check(parts, want, [k for k in cols if k != "filter"])


@pytest.mark.parametrize("rpp", [16384, 131072])
def test_bad_page(rpp):
    cols = _edge_columns(rpp * 2)
    t = paged.PagedTable.from_columns(cols, rows_per_page=rpp)
    pages = t.pages.clone().pin_memory()
    pages[int(t.directory[1])] ^= 0xFF
    bad = paged.PagedTable(pages, t.directory, t.n_rows, t.rows_per_page, t.names, t.esizes)
    parts = paged.paged_scan(bad, "filter", -(1 << 62), 1 << 62, "key", B=8, groups_per_batch=2)
    torch.cuda.synchronize()
    s = parts.read_stats()
    assert s["bad_pages"] == 4 and s["rows"] == rpp
