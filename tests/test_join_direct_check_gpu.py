"""When the direct join (csrc/join_direct.cu) may take its packed sums: rows
without a group neither hide a sum that left its field nor cost a second run."""
import numpy as np
import pytest
import torch

import oracle
from pageflow_b200 import _native
from pageflow_b200.join_aggregate import JoinAggregate

pytestmark = pytest.mark.gpu

# kernel launches of one attempt (init, build, probe, finish)
ATTEMPT = 4


@pytest.fixture(autouse=True)
def _no_overrides(monkeypatch):
    for v in ("PF_JOIN_PATH", "PF_SJ_FP", "PF_SJ_TARGET", "PF_COUNTED"):
        monkeypatch.delenv(v, raising=False)


def _run(bkey, bgrp, fk, price, G):
    """The plan's launches; its results held against the oracle."""
    args = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (bkey, bgrp, fk, price)]
    s, c, matched, _ = oracle.join_aggregate(bkey, bgrp, fk, price, None, 100, 0, G, B=16)
    plan = JoinAggregate(len(bkey), len(fk), 0, G, "cuda", autotune=False)
    assert plan.direct
    L = _native.lib()
    before = L.pf_launch_count()
    keys, sums, counts = plan.run(*args)
    launches = L.pf_launch_count() - before
    here = np.nonzero(c)[0]
    assert np.array_equal(keys.cpu().numpy(), here)
    assert np.array_equal(sums.cpu().numpy(), s[here])
    assert np.array_equal(counts.cpu().numpy(), c[here])
    assert plan.read_stats().matched == matched
    return launches


@pytest.mark.parametrize("outside", [1, 2, 5])
@pytest.mark.parametrize("overflows", [0, 1, 2])
def test_rows_without_a_group_hide_no_overflow(outside, overflows):
    """90,000 probe rows into 3,000 groups: values of 2^55 - 1 and 1 in one
    group make its sum 2^55 while a count field holds nine bits, and a matched
    row of a group out of range is in no packed word."""
    n, G = 90_000, 3000
    bkey = np.arange(1, 6001, dtype=np.int64)
    bgrp = (np.arange(6000) % G).astype(np.int32)
    bgrp[5990:] = G + 7
    fk = np.full(n, 10**9, np.int64)      # no build row
    price = np.zeros(n, np.int64)
    for k in range(overflows):
        fk[2 * k:2 * k + 2] = 5 + k + 1   # group 5 + k
        price[2 * k] = (1 << 55) - 1
        price[2 * k + 1] = 1
    fk[1000:1000 + outside] = bkey[5990:5990 + outside]
    price[1000:1000 + outside] = 3
    _run(bkey, bgrp, fk, price, G)


def test_rows_without_a_group_cost_no_second_run():
    rng = np.random.default_rng(2)
    bkey = rng.permutation(20_000).astype(np.int64)
    bgrp = rng.integers(0, 4000, 20_000).astype(np.int32)
    bgrp[::100] = 4000
    bgrp[1] = -1
    fk = rng.integers(0, 22_000, 200_000)
    assert _run(bkey, bgrp, fk, rng.integers(0, 1 << 24, 200_000), 4000) == ATTEMPT


def _groups(kind, n, G, rng):
    g = rng.integers(0, G, n)
    if kind == "zipf":
        w = 1.0 / np.arange(1, G + 1)
        g = np.searchsorted(np.cumsum(w) / w.sum(), rng.random(n)).clip(max=G - 1)
    elif kind != "equal":
        g[rng.random(n) < float(kind)] = 7
    return g.astype(np.int32)


@pytest.mark.parametrize("kind", ["equal", "zipf", "0.002", "0.01", "0.1", "0.6"])
@pytest.mark.parametrize("np_", [60_000, 900_001, 4_000_000])
def test_skewed_groups_cost_no_second_run(kind, np_):
    rng = np.random.default_rng(np_)
    nb, G = 150_001, 5000
    fk = rng.integers(0, nb + nb // 10, np_)
    assert _run(rng.permutation(nb).astype(np.int64), _groups(kind, nb, G, rng), fk,
                rng.integers(0, 1 << 24, np_), G) == ATTEMPT


@pytest.mark.parametrize("np_", [900_001, 4_000_000])
def test_skewed_keys_cost_no_second_run(np_):
    rng = np.random.default_rng(np_)
    nb, G = 150_001, 5000
    fk = (rng.random(np_) ** 40 * nb).astype(np.int64)
    assert _run(rng.permutation(nb).astype(np.int64), _groups("equal", nb, G, rng), fk,
                rng.integers(0, 1 << 24, np_), G) == ATTEMPT


@pytest.mark.parametrize("lo,hi", [(-1000, 1000), (-5, 0), (-(1 << 63), (1 << 63) - 1),
                                   (1 << 55, 1 << 60)])
@pytest.mark.parametrize("every", [1, 1000])
@pytest.mark.parametrize("np_", [200_000, 4_000_000])
def test_values_outside_a_packed_words_cost_no_second_run(lo, hi, every, np_):
    rng = np.random.default_rng(5)
    nb, G = 20_001, 3000
    price = rng.integers(0, 1 << 24, np_)
    price[::every] = rng.integers(lo, hi, len(price[::every]), endpoint=True)
    assert _run(rng.permutation(nb).astype(np.int64), _groups("equal", nb, G, rng),
                rng.integers(0, nb, np_), price, G) == ATTEMPT
