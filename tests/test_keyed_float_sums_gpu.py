"""The one-read pass's float64 sums against exact ones (math.fsum): with the
adds' rounding errors given back, a sum of n values is off by its own rounding,
half an ulp, and by the errors' own, at most (n eps)^2 of the values' sizes."""
import math

import numpy as np
import pytest
import torch

from pageflow_b200.keyed_aggregate import KeyedPass1

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def _values(kind, n, rng):
    if kind == "prices":
        return rng.integers(90_000, 10_500_001, n) / 100
    if kind == "normal":
        return rng.standard_normal(n)
    v = rng.standard_normal(n)   # large ones that cancel
    v[::3] += 1e15
    v[1::3] -= 1e15
    return v


def _pass1(key, v, aggs, B=1):
    p = KeyedPass1([0], aggs)
    p._hash_and_sort = None   # the one-read route, or an error
    out, _ = p.pass1({0: torch.from_numpy(key).cuda(), 1: torch.from_numpy(v).cuda()}, B)
    return [t.cpu().numpy() for t in out[1:]]


@pytest.mark.parametrize("kind", ["prices", "normal", "cancel"])
@pytest.mark.parametrize("n,groups", [(300_001, 3), (300_001, 150), (300_001, 20_011), (1_000_003, 90_001),
                                      (33, 5), (1, 1)])
def test_sums_are_exact_to_their_own_rounding(kind, n, groups):
    rng = np.random.default_rng(n + groups)
    key, v = rng.integers(0, groups, n), _values(kind, n, rng)
    k, s, avg, c = _pass1(key, v, [("sum", 1), ("avg", 1), ("count", None)])
    order = np.argsort(key, kind="stable")
    ends = np.cumsum(np.bincount(key, minlength=groups))
    for i in range(0, len(k), max(1, len(k) // 3000)):
        x = v[order[ends[k[i]] - c[i]:ends[k[i]]]]
        want = math.fsum(x)
        bound = EPS * abs(want) + (len(x) * EPS) ** 2 * np.abs(x).sum()
        assert abs(s[i] - want) <= bound
        assert avg[i, 0] == s[i] and avg[i, 1] == len(x) == c[i]


@pytest.mark.parametrize("copies", [1, 4000])
def test_infinities_nans_and_overflow(copies):
    """Small groups and ones that a block folds in its own table first."""
    inf, nan, big = math.inf, math.nan, 1.7e308
    rows = [[inf, 1.0], [-inf, 2.0], [inf, -inf], [nan, 1.0], [big, big], [-big, -big], [1e300, -1e300],
            [-64.0, 64.0], [5e-324, 5e-324], [0.0, -0.0]]
    key = np.repeat(np.arange(len(rows)), 2)
    v = np.array(rows).ravel()
    more = np.zeros(len(rows) * copies)
    k, s, avg = _pass1(np.concatenate([key, np.tile(np.arange(len(rows)), copies)]),
                       np.concatenate([v, more]), [("sum", 1), ("avg", 1)])
    want = np.array([inf, -inf, nan, nan, inf, -inf, 0.0, 0.0, 1e-323, 0.0])[k]
    assert np.array_equal(s, want, equal_nan=True)
    assert np.array_equal(avg[:, 0], want, equal_nan=True)
    assert (avg[:, 1] == copies + 2 - (k == 7)).all()


def test_a_float32_column_and_many_float64_ones():
    """float32 sums are added in float64 as they are; more float64 sums than the
    table has accumulators for go the general way."""
    rng = np.random.default_rng(1)
    n = 60_000
    key = rng.integers(0, 50, n)
    v = rng.standard_normal(n).astype(np.float32)
    k, s = _pass1(key, v, [("sum", 1)])
    want = np.bincount(key, v.astype(np.float64), 50)
    # within a rounding to float32 and n adds in float64
    assert np.all(np.abs(s - want[k]) <= 2.0 ** -24 * np.abs(want[k]) + n * EPS * np.abs(v).sum())
    cols = {0: torch.from_numpy(key).cuda()}
    for c in range(1, 9):
        cols[c] = torch.from_numpy(rng.integers(0, 1000, n).astype(np.float64)).cuda()
    p = KeyedPass1([0], [("sum", c) for c in range(1, 9)])
    out, _ = p.pass1(cols)
    for c in range(1, 9):
        want = np.bincount(key, cols[c].cpu().numpy(), 50)
        assert np.array_equal(out[1 + c].cpu().numpy(), want[out[1].cpu().numpy()])
