"""The join without a radix pass (csrc/join_direct.cu) against the oracle: the
sums' three forms and the line between them (2048 groups), the table at its
fullest, rows past their home bucket, extreme keys, skewed keys, values that
leave the packed sum's field, groups outside the range, and hashes that crowd
the table (the radix path then gives the result)."""
import numpy as np
import pytest
import torch

import oracle
from pageflow_b200 import _native
from pageflow_b200.join_aggregate import JoinAggregate, join_group_aggregate

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _no_overrides(monkeypatch):
    for v in ("PF_JOIN_PATH", "PF_SJ_FP", "PF_SJ_TARGET", "PF_COUNTED"):
        monkeypatch.delenv(v, raising=False)


def _check(bkey, bgrp, fk, price, disc, gmin, G, direct=True):
    args = [None if x is None else torch.from_numpy(np.ascontiguousarray(x)).cuda()
            for x in (bkey, bgrp, fk, price, disc)]
    s, c, matched, _ = oracle.join_aggregate(bkey, bgrp, fk, price, disc, 100, gmin, G, B=16)
    here = np.nonzero(c)[0]
    plan = JoinAggregate(len(bkey), len(fk), gmin, G, "cuda", autotune=False)
    assert plan.direct == direct
    for _ in range(2):   # a plan runs again
        keys, sums, counts = plan.run(*args)
        assert np.array_equal(keys.cpu().numpy(), gmin + here)
        assert np.array_equal(sums.cpu().numpy(), s[here])
        assert np.array_equal(counts.cpu().numpy(), c[here])
        assert np.array_equal(plan.sum.cpu().numpy(), s)
        assert np.array_equal(plan.count.cpu().numpy(), c)
        assert plan.read_stats().matched == matched
    plan.sum.fill_(-1)
    plan.aggregate(*args)
    assert np.array_equal(plan.sum.cpu().numpy(), s)
    k2, s2, c2 = plan.finish()
    assert torch.equal(k2, keys) and torch.equal(s2, sums) and torch.equal(c2, counts)
    return plan


def _inputs(nb, np_, G, seed=0, disc=True, skew=1.0):
    rng = np.random.default_rng(seed)
    bkey = rng.permutation(np.unique(rng.integers(-(1 << 62), 1 << 62, nb + 9)))[:nb]
    bgrp = rng.integers(0, G, nb).astype(np.int32)
    at = np.minimum((rng.random(np_) ** skew * nb).astype(np.int64), nb - 1)
    fk = np.where(rng.random(np_) < 0.9, bkey[at], rng.integers(0, 1 << 62, np_))
    price = rng.integers(90_000, 10_500_001, np_)
    return bkey, bgrp, fk, price, rng.integers(0, 11, np_) if disc else None


@pytest.mark.parametrize("G", [1, 2, 25, 64, 65, 1024, 2047, 2048, 2049, 4096, 4097, 12_289])
@pytest.mark.parametrize("disc", [True, False])
def test_group_counts_at_the_lines_between_the_sums_forms(G, disc):
    bkey, bgrp, fk, price, d = _inputs(30_011, 70_003, G, G, disc)
    _check(bkey, bgrp - 5, fk, price, d, -5, G)


@pytest.mark.parametrize("nb,np_", [(1, 1), (2, 513), (255, 1), (257, 511), (1023, 512), (1024, 513)])
def test_the_smallest_sizes(nb, np_):
    _check(*_inputs(nb, np_, 3, nb), 0, 3)


@pytest.mark.parametrize("nb", [76, 77, 19_660, 19_661, 78_643, 78_644])
def test_tables_at_their_fullest_and_one_row_past(nb):
    """0.3 of 4 * 2^q entries: some rows lie past their home bucket."""
    _check(*_inputs(nb, 150_001, 900, nb), 0, 900)


def test_extreme_keys_values_and_discounts():
    I = np.iinfo(np.int64)
    bkey = np.array([I.min, I.max, 0, -1, 5, I.min + 1, 1 << 40], np.int64)
    bgrp = np.array([0, 1, 2, 3, 4, 5, 6], np.int32)
    fk = np.array([I.min, I.min, I.max, 7, -1, I.min + 1, 0, I.min, 1 << 40], np.int64)
    price = np.array([I.max, 5, -7, 1, -(1 << 50), 3, 1 << 61, -1, 9], np.int64)
    for d in (None, np.array([0, 300, -4, 1, 2, 100, 101, 0, 99], np.int64)):
        _check(bkey, bgrp, fk, price, d, 0, 7)
        _check(bkey, bgrp, fk, price, d, 0, 5000)


@pytest.mark.parametrize("top", [1 << 30, 1 << 52, 1 << 60, -5])
def test_values_that_leave_the_packed_sums_field(top):
    """A field of 2^(64 - count bits): values past it, sums past it, and
    negative ones are summed in two words."""
    bkey, bgrp, fk, price, _ = _inputs(20_000, 90_000, 3000, 3)
    price = price.copy()
    price[::1000] = top
    _check(bkey, bgrp, fk, price, None, 0, 3000)


@pytest.mark.parametrize("skew", [4, 30])
@pytest.mark.parametrize("G", [700, 30_000])
def test_skewed_keys(G, skew):
    _check(*_inputs(40_000, 400_000, G, skew, skew=skew), 0, G)


def test_one_group_takes_every_row():
    """A count past the packed field's (256 times the mean) and a hot cache."""
    bkey, bgrp, fk, price, d = _inputs(10_000, 300_000, 5000, 4)
    bgrp[:] = 77
    _check(bkey, bgrp, fk, price, d, 0, 5000)


@pytest.mark.parametrize("nb,np_,G", [(1_250_000, 2_000_000, 40), (2_600_000, 3_000_000, 200_000),
                                      (3_400_000, 2_000_000, 9_000)])
def test_the_large_tables(nb, np_, G):
    """32, 64 and 128 MiB, the last two up to 0.4 full."""
    _check(*_inputs(nb, np_, G, nb), 0, G)


def test_groups_outside_the_range_are_counted_and_left_out():
    bkey, bgrp, fk, price, d = _inputs(5_000, 20_000, 100, 6)
    bgrp[::3] = 100 + bgrp[::3]
    bgrp[1] = -1
    for G in (100, 3000):
        plan = _check(bkey, bgrp, fk, price, d, 0, G)
        bad = int(((bgrp < 0) | (bgrp >= G)).sum())
        assert plan.read_stats().bad_groups == bad


def test_keys_of_one_radix_bucket():
    """Hashes that share their top nine bits spread over the table."""
    rng = np.random.default_rng(8)
    k = rng.integers(0, 1 << 62, 4_000_000)
    k = np.unique(k[(oracle.mix64(k).view(np.uint64) >> np.uint64(55)) == 3])
    bkey = rng.permutation(k)
    n = len(bkey)
    fk = bkey[rng.integers(0, n, 5 * n)]
    _check(bkey, rng.integers(0, 50, n).astype(np.int32), fk, rng.integers(0, 1000, 5 * n), None,
           0, 50)


def test_hashes_that_crowd_the_table_take_the_radix_path():
    """Keys whose rotated hashes share their top 21 bits: one home bucket."""
    rng = np.random.default_rng(9)
    n = 2000
    rot = (np.uint64(5) << np.uint64(43)) | rng.integers(0, 1 << 43, n, dtype=np.uint64)
    h = np.unique((rot >> np.uint64(21)) | (rot << np.uint64(43)))
    k = h.copy()
    with np.errstate(over="ignore"):
        for c in (0xc4ceb9fe1a85ec53, 0xff51afd7ed558ccd):
            k ^= k >> np.uint64(33)
            k *= np.uint64(pow(c, -1, 1 << 64))
        k ^= k >> np.uint64(33)
    bkey = k.view(np.int64)
    assert np.array_equal(oracle.mix64(bkey).view(np.uint64), h)
    m = len(bkey)
    fk = bkey[rng.integers(0, m, 9000)]
    _check(bkey, rng.integers(0, 20, m).astype(np.int32), fk, rng.integers(0, 1000, 9000), None,
           0, 20)


def test_what_keeps_the_radix_path():
    """A fan-out, knobs or an override; a build past the table; groups whose
    numbers leave the entry no room."""
    assert not JoinAggregate(1000, 1000, 0, 10, "cuda", B=4).direct
    assert not JoinAggregate(1000, 1000, 0, 10, "cuda", knobs=dict(path=0, table=0)).direct
    L = _native.lib()
    assert L.pf_join_direct_fits(6_710_886, 10, 1000) == 1
    assert L.pf_join_direct_fits(6_710_887, 10, 1000) == 0
    assert L.pf_join_direct_fits(1000, 10, (1 << 19) - 2) == 1
    assert L.pf_join_direct_fits(1000, 10, (1 << 19) - 1) == 0
    assert L.pf_join_direct_fits(0, 10, 10) == 0


def test_the_autotuned_plan_and_the_one_shot_call(tmp_path, monkeypatch):
    monkeypatch.setenv("PAGEFLOW_TUNE_CACHE", str(tmp_path / "tune.json"))
    bkey, bgrp, fk, price, d = _inputs(9_000, 40_000, 37, 11)
    t = [torch.from_numpy(x).cuda() for x in (bkey, bgrp, fk, price, d)]
    s, c, _, _ = oracle.join_aggregate(bkey, bgrp, fk, price, d, 100, 0, 37, B=16)
    keys, sums, counts = join_group_aggregate(*t)
    assert np.array_equal(sums.cpu().numpy(), s[keys.cpu().numpy()])
    assert np.array_equal(counts.cpu().numpy(), c[keys.cpu().numpy()])
