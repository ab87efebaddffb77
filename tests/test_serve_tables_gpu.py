"""Dimension tables of every form and groups of every kind of sum: requests
against the oracle, whole numbers equal."""
import ctypes
import dataclasses

import numpy as np
import pytest
import torch

import oracle
from pageflow_b200 import serve
from pageflow_b200._native import check, lib, ptr, stream_of
from tests.test_aggregate_gpu import _unmix64_array

pytestmark = pytest.mark.gpu


def _crowded(n):
    """Keys whose hashes share a compact table's home bucket (its hash is
    mix64's bits rotated by 21)."""
    h = (np.uint64(5) << np.uint64(45)) | np.arange(n, dtype=np.uint64) << np.uint64(3)
    rot = (h >> np.uint64(21)) | (h << np.uint64(43))
    return _unmix64_array(rot)


@pytest.mark.parametrize("nk,ng,kind,skew", [
    (1, 1, "plain", 0),                 # the smallest table
    (129, 3, "plain", 0),               # own cells, many copies a group
    (5000, 512, "plain", 0),            # the most groups kept in own cells
    (5000, 513, "plain", 1.2),          # the first of the others, with hot groups
    (70_001, 4096, "plain", 0),         # no group comes again: straight to the slab
    (70_001, 20_000, "plain", 1.5),
    (3000, 2_000_000, "plain", 0),      # no room for the group: 16-byte slots
    (3000, 40, "crowded", 0),           # a compact table's run full: built again
    (3000, 40, "unaligned", 0),         # a table on 16 bytes
])
def test_table_forms_and_sums(nk, ng, kind, skew):
    dev = torch.device("cuda", 0)
    n = 120_011
    spec = dataclasses.replace(serve.scaled(serve.SERVE, 20_000), dim_keys=(nk,),
                               dim_groups=(ng,), fact_rows=n, n_ranks=max(nk, 1000),
                               probe_min=1, probe_max=n)
    rng = np.random.default_rng(nk + ng)
    keys = _crowded(nk) if kind == "crowded" else rng.choice(1 << 40, nk, replace=False) - (1 << 39)
    if nk > 2:
        keys[0], keys[1], keys[2] = -1, 0, np.iinfo(np.int64).min
    keys = keys.astype(np.int64)
    groups = rng.integers(0, ng, nk).astype(np.int32)
    if nk > 2:
        groups[0], groups[1] = 0, ng - 1
    pick = (np.minimum(rng.zipf(skew, n) - 1, nk - 1) if skew else rng.integers(0, nk, n))
    fk = keys[pick]
    miss = rng.random(n) < 0.3
    fk[miss] = rng.integers(1 << 50, 1 << 60, miss.sum())
    date = rng.integers(0, 100, n).astype(np.int32)
    value = rng.integers(-(1 << 62), 1 << 62, n)      # sums wrap at 64 bits

    dims = serve.Dimensions(spec, dev)
    fact = serve.FactPool(spec, dev)
    for d, h in ((fact.fk, fk), (fact.date, date), (fact.value, value),
                 (dims.keys[0], keys), (dims.groups[0], groups)):
        d.copy_(torch.from_numpy(h))
    L = lib()
    tb = L.pf_dim_table_bytes(nk)
    off = 16 if kind == "unaligned" else 0
    t = torch.full((tb + off,), 255, dtype=torch.uint8, device=dev)[off:]
    stats = torch.empty(2, dtype=torch.int64, device=dev)
    check(L.pf_dim_build(ptr(dims.keys[0]), ptr(dims.groups[0]), nk, ng, ptr(t), tb, ptr(stats),
                         stream_of(dev)), "dim_build")
    assert stats.tolist() == [0, 0]
    dims.tables[0] = t

    reqs = [serve.Request(0, 0, 0, n, 10, 90), serve.Request(1, 0, 7, n - 7, 0, 100),
            serve.Request(2, 0, n - 1, 1, 0, 100), serve.Request(3, 0, 0, 5000, 50, 51),
            serve.Request(4, 0, 100, 70_000, 200, 300)]
    srv = serve.Server(dims, fact, 1 << 30, dev, iter_rows=1 << 16, pinned_bytes=1 << 28)
    srv.run(reqs, timeout_s=60)
    for r in reqs:
        s = slice(r.row0, r.row0 + r.n_rows)
        want = oracle.serve_request(keys, groups, ng, fk[s], date[s], value[s], r.date_lo,
                                    r.date_hi)
        for a, b in zip(r.result, want):
            assert np.array_equal(a, b), r.id


def test_groups_outside_are_counted_once():
    """A key whose group is out of range matches without a group, in both
    forms of table; a crowded one counts it once."""
    dev = torch.device("cuda", 0)
    L = lib()
    for keys in (np.arange(3000), _crowded(3000)):
        k = torch.from_numpy(np.ascontiguousarray(keys, np.int64)).to(dev)
        g = torch.arange(3000, dtype=torch.int32, device=dev) - 5
        tb = L.pf_dim_table_bytes(3000)
        t = torch.empty(tb, dtype=torch.uint8, device=dev)
        stats = torch.empty(2, dtype=torch.int64, device=dev)
        check(L.pf_dim_build(ptr(k), ptr(g), 3000, 2990, ptr(t), tb, ptr(stats),
                             stream_of(dev)), "dim_build")
        assert stats.tolist() == [10, 0]


def test_slabs_are_cleared_and_their_neighbours_kept():
    """More slabs than one launch takes, of sizes around a block's and a grid's
    share, each with a guard pair behind it."""
    dev = torch.device("cuda", 0)
    L = lib()
    sizes = [1, 2, 255, 256, 257, 1023, 1025, 40_000] * 33
    ends = np.cumsum([s + 1 for s in sizes])
    pool = torch.full((int(ends[-1]), 2), -1, dtype=torch.int64, device=dev)
    starts = ends - np.array(sizes) - 1
    at = (ctypes.c_void_p * len(sizes))(*[pool.data_ptr() + 16 * int(a) for a in starts])
    ng = (ctypes.c_int64 * len(sizes))(*sizes)
    check(L.pf_serve_clear(at, ng, len(sizes), stream_of(dev)), "serve_clear")
    want = np.zeros((int(ends[-1]), 2), np.int64)
    want[ends - 1] = -1
    assert np.array_equal(pool.cpu().numpy(), want)
