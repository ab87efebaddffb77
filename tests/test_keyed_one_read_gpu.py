"""Pass 1 of the keyed aggregation in one read of its rows (csrc/keyed.cu)
against the general route, hash then radix sort then a reduction a column
(KeyedPass1._hash_and_sort): every column type, width and aggregate that it
takes, one group to as many as its table holds, hashes at the edges of the
int64 range and crowded into one bucket of it; and the in-place fold of a
sorted run (pf_fold_sorted_run) against numpy.

Integers are equal; a float64 sum of at most 64K terms, added in any order,
is within 64K * 2^-53 of the sum of their magnitudes (7.3e-12 relative)."""
import numpy as np
import pytest
import torch

from pageflow_b200 import keyed_aggregate as ka
from pageflow_b200 import sorted_run_merge as srm

pytestmark = pytest.mark.gpu
ALL = [('sum', 10), ('count', None), ('count', 10), ('avg', 10), ('min', 11), ('max', 11),
       ('sum', 11), ('sum', 12), ('avg', 12), ('sum', 13), ('avg', 13), ('min', 10),
       ('max', 10)]


def _cols(n, keys, seed=0):
    rng = np.random.default_rng(seed)
    c = {i + 1: torch.from_numpy(k).cuda() for i, k in enumerate(keys)}
    v = rng.integers(-10**12, 10**12, n)
    v[::7] = -64                                   # the null
    w = rng.integers(-100, 100, n).astype(np.int32)
    f = rng.random(n) * 1e6
    f[::5] = -64.0
    c.update({10: torch.from_numpy(v).cuda(), 11: torch.from_numpy(w).cuda(),
              12: torch.from_numpy(f).cuda(),
              13: torch.from_numpy(rng.integers(0, 1 << 10, n).astype(np.float32)).cuda()})
    return c


def _compare(cols, key_ids, aggs, coeffs=None, emitted=None):
    p = ka.KeyedPass1(key_ids, aggs, emitted)
    keys = [ka._as_2d(cols[k]) for k in key_ids]
    p._coeffs = ka.make_key_coeffs(keys, keys[0].device) if coeffs is None else coeffs
    # the general route adds float32 columns in float32, whose sums of these
    # whole numbers pass 2^24: their oracle is its sum of the same column as
    # float64, exact here, rounded once
    wide = {c: v.double() if c == 13 else v for c, v in cols.items()}
    got, want = p._one_read(cols, keys, 16), p._hash_and_sort(wide, keys)
    assert got is not None
    got, buckets = got
    bucket, counts, counts_t = ka.hash_buckets(want[0], 16)
    assert torch.equal(buckets[0], bucket) and torch.equal(buckets[2], counts_t)
    assert buckets[1] == counts
    want = [w.to(g.dtype) if w.is_floating_point() else w for g, w in zip(got, want)]
    assert len(got) == len(want)
    for g, w in zip(got, want):
        assert g.dtype == w.dtype and g.shape == w.shape
        if g.dtype.is_floating_point:
            scale = w.abs().clamp_min(1.0)
            assert float(((g - w).abs() / scale).max()) <= 7.3e-12
        else:
            assert torch.equal(g, w)
    return got


@pytest.mark.parametrize("groups", [1, 2, 3, 17, 500, 513, 5000, 60_000])
def test_group_counts(groups):
    n = 60_001
    rng = np.random.default_rng(groups)
    keys = [rng.integers(0, groups, n) - groups // 2]
    _compare(_cols(n, keys), [1], ALL[:8])
    _compare(_cols(n, keys), [1], ALL[8:])


@pytest.mark.parametrize("n", [1, 31, 1023, 1024, 1025, 4097])
def test_row_counts_at_the_edges_of_a_tile(n):
    rng = np.random.default_rng(n)
    keys = [rng.integers(0, 9, n), rng.integers(-3, 3, n).astype(np.int32)]
    _compare(_cols(n, keys), [1, 2], ALL[:7])
    _compare(_cols(n, keys), [1, 2], [], emitted=[2])


@pytest.mark.parametrize("dtype", [np.int8, np.int16, np.int32, np.int64, np.float32, np.float64])
@pytest.mark.parametrize("width", [0, 1, 2, 3, 5])
def test_key_types_and_widths(dtype, width):
    n = 5_003
    rng = np.random.default_rng(width)
    keys = [rng.integers(-2, 3, (n, width) if width else n).astype(dtype),
            rng.integers(0, 5, n)]
    cols = _cols(n, keys)
    _compare(cols, [1, 2], [('count', None), ('sum', 10)])
    # a column that starts off its natural alignment of 8 bytes
    cols[1] = cols[1][1:]
    cols[2] = cols[2][1:]
    cols[10] = cols[10][1:]
    _compare(cols, [2, 1], [('sum', 10)])


def test_the_hash_that_marks_an_empty_slot():
    """INT64_MIN (an odd coefficient keeps it) among other keys, and alone."""
    lo = np.iinfo(np.int64).min
    for keys in (np.array([lo, 5, lo, 7, lo, 5]), np.full(300, lo)):
        n = keys.shape[0]
        got = _compare(_cols(n, [keys]), [1], ALL[:7],
                       [torch.tensor([3], dtype=torch.int64, device="cuda")])
        assert int(got[0][0]) == lo


def test_hashes_crowded_into_one_bucket():
    """5000 neighbouring keys and one at the far end of the range."""
    n = 40_000
    keys = np.random.default_rng(2).integers(0, 5000, n)
    keys[17] = 1 << 40
    _compare(_cols(n, [keys]), [1], ALL[:7],
             [torch.tensor([1], dtype=torch.int64, device="cuda")])


@pytest.mark.parametrize("share", [1, 3])
def test_more_groups_than_the_first_table_holds(share):
    """3M rows of single groups take the general route, 1M groups of three
    rows a second table sized by the first one's estimate."""
    n = 3_000_000
    key = torch.randperm(n, device="cuda") // share
    cols = {1: key, 10: key * 3 - 64, 11: key.to(torch.int32)}
    aggs = ALL[:7]
    p = ka.KeyedPass1([1], aggs)
    p._coeffs = ka.make_key_coeffs([key[:, None]], "cuda")
    got = p._one_read(cols, [key[:, None]], 1)
    assert (got is None) == (share == 1)
    out, _ = p.pass1(cols)
    want = p._hash_and_sort(cols, [key[:, None]])
    assert out[0].numel() == n // share
    for g, w in zip(out, want):
        assert g.dtype == w.dtype and torch.equal(g, w)


def test_what_the_slots_do_not_hold_takes_the_general_route():
    n = 1000
    cols = _cols(n, [np.arange(n) % 7])
    cols[14] = cols[11].to(torch.int16)
    cols[15] = torch.stack([cols[10], cols[10]], dim=1)
    for aggs in ([('min', 12)], [('max', 13)], [('sum', 14)]):
        p = ka.KeyedPass1([1], aggs)
        keys = [cols[1][:, None]]
        p._coeffs = ka.make_key_coeffs(keys, "cuda")
        assert p._one_read(cols, keys) is None
        assert p.pass1(cols)[0][0].numel() == 7


@pytest.mark.parametrize("tick", ["all", "one", "some_new"])
@pytest.mark.parametrize("n", [1, 255, 257, 70_000])
def test_a_tick_folded_into_its_run(n, tick):
    rng = np.random.default_rng(n)
    run = np.sort(rng.choice(4 * n, n, replace=False)).astype(np.int64)
    tk = run[::3] if tick == "all" else run[-1:]
    if tick == "some_new":
        tk = np.unique(np.concatenate([run[::2], run[::5] + 1]))
    vals = [rng.integers(-99, 99, n), rng.random((n, 2)), rng.integers(-9, 9, n).astype(np.int32)]
    tv = [rng.integers(-99, 99, tk.size), rng.random((tk.size, 2)),
          rng.integers(-9, 9, tk.size).astype(np.int32)]
    ops = ["sum", "sum", "amax"]
    room = n + tk.size + 3
    kb = torch.zeros(room, dtype=torch.int64, device="cuda")
    vb = [torch.zeros((room,) + v.shape[1:], dtype=torch.from_numpy(v).dtype, device="cuda")
          for v in vals]
    # an empty run takes the first tick whole
    m = srm.merge_sorted_unique_runs_inplace(kb, vb, 0, torch.from_numpy(run).cuda(),
                                             [torch.from_numpy(v).cuda() for v in vals], ops)
    m = srm.merge_sorted_unique_runs_inplace(kb, vb, m, torch.from_numpy(tk).cuda(),
                                             [torch.from_numpy(v).cuda() for v in tv], ops)
    keys = np.union1d(run, tk)
    assert m == keys.size and np.array_equal(kb[:m].cpu().numpy(), keys)
    for b, v, t, op in zip(vb, vals, tv, ops):
        want = np.zeros((m,) + v.shape[1:], v.dtype)
        at, ta = np.searchsorted(keys, run), np.searchsorted(keys, tk)
        fresh = ~np.isin(tk, run)
        want[at] = v
        want[ta[fresh]] = t[fresh]
        old = want[ta[~fresh]]
        want[ta[~fresh]] = old + t[~fresh] if op == "sum" else np.maximum(old, t[~fresh])
        assert np.array_equal(b[:m].cpu().numpy(), want)
    assert int(kb[m:].abs().sum()) == 0
