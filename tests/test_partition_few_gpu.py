"""Few buckets: every bucket count a warp stages by itself and the first it
does not, every word width, masks and both prologues, sizes around a warp's
segment and a tile, against the oracle, bit for bit."""
import pytest
import torch

from tests.dropin import partition
from tests.test_partition_gpu import _check, _contradicted, _mask, _table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("keep,select_first", [(None, False), (0.03, True), (0.4, False),
                                               (0.9, True), (1.0, False)])
def test_widths_and_masks(B, keep, select_first):
    n = 50_021
    cols = _table(n, ["i8", "i32", "i16", "i64"], seed=B, key_pos=2)
    mask = None if keep is None else _mask(n, keep, seed=B + 7)
    _check(cols, 2, mask, 6_000_000_007, B, compact=[False] * 5, count=keep is not None,
           select_first=select_first)


@pytest.mark.parametrize("n", [0, 1, 31, 255, 256, 257, 2047, 2048, 2049, 4097])
@pytest.mark.parametrize("masked", [False, True])
def test_sizes(n, masked):
    mask = _mask(n, 0.5, seed=n) if masked else None
    _check(_table(n, ["i32", "i8"], seed=n), 0, mask, 3, 8, compact=[False] * 3, count=masked,
           select_first=False)


@pytest.mark.parametrize("B", [2, 16])
def test_one_bucket_holds_every_row(B):
    _check(_table(9_001, ["i64", "i8"], seed=5, skew=True), 0, None, 0, B)


@pytest.mark.parametrize("offset", [1, 3])
def test_columns_off_their_words(offset):
    """Views whose narrow columns start off a word's boundary keep the general
    kernel's copies."""
    cols = [c[offset:] for c in _table(30_000, ["i32", "i16", "u8x8", "u8x3"], seed=9)]
    _check(cols, 0, None, 0, 8)


@pytest.mark.parametrize("select_first", [False, True])
@pytest.mark.parametrize("off", [-37, 41])
def test_a_contradicted_count_writes_nothing_past_it(select_first, off):
    n = 60_003
    cols = _table(n, ["i64", "i8"], seed=91)
    mask = _mask(n, 0.2, seed=92)
    wrong = int(mask.sum()) + off
    call = partition(list(cols), 0, mask, 0, 8, n_valid=wrong, select_first=select_first)
    torch.cuda.synchronize()
    assert _contradicted(call, wrong)
    _check(cols, 0, mask, 0, 8, compact=[False] * 3, count=True, select_first=select_first)
