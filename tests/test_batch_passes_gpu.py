"""The batch engine's two passes (csrc/batch.cu) against the oracle: compact
tables and the sizes where they end (groups numbered past the rows), packed
sums and the values and skews that leave their fields (those instances are run
again in the same call, and from the start in later ones), hashes that crowd a
compact table, and mixes of all of them in one batch, run and replayed."""
import numpy as np
import pytest
import torch

import oracle
from pageflow_b200.batch import BatchJoinAggregate, Instance

pytestmark = pytest.mark.gpu


def _instance(nb, np_, G, seed, values=(0, 1 << 24), skew=1.0, gmin=0):
    rng = np.random.default_rng(seed)
    key = rng.permutation(np.unique(rng.integers(-(1 << 62), 1 << 62, nb + 9)))[:nb]
    grp = (rng.integers(0, G, nb) + gmin).astype(np.int32)
    at = np.minimum((rng.random(np_) ** skew * nb).astype(np.int64), nb - 1)
    fk = np.where(rng.random(np_) < 0.9, key[at], rng.integers(0, 1 << 62, np_))
    return key, grp, fk, rng.integers(values[0], values[1], np_), gmin, G


def _run_and_check(cases, runs=3, graph=False):
    insts = [Instance(*[torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in c[:4]], *c[4:])
             for c in cases]
    b = BatchJoinAggregate(insts, "cuda")
    g = b.graph() if graph else None
    want = [oracle.join_aggregate(c[0], c[1], c[2], c[3], None, 0, c[4], c[5], B=4) for c in cases]
    for _ in range(runs):
        g.replay() if graph else b.run()
        torch.cuda.synchronize()
        for i, (s, c, _, _) in enumerate(want):
            gs, gc = b.result(i)
            assert np.array_equal(gc.cpu().numpy(), c), f"instance {i} counts"
            assert np.array_equal(gs.cpu().numpy(), s), f"instance {i} sums"
        st = b.read_stats()
        assert st["matched"] == sum(w[2] for w in want)
        assert st["device_error"] == 0 and st["overflow"] == 0
        bad = sum(int(((c[1] < c[4]) | (c[1] >= c[4] + c[5])).sum()) for c in cases)
        assert st["bad_groups"] == bad


@pytest.mark.parametrize("nb,np_,G", [(1, 1, 1), (1, 600, 1), (4096, 16384, 2), (4097, 16385, 4095),
                                      (4095, 16383, 4096), (60_000, 70_001, 4097),
                                      (1000, 40_000, 1000), (1000, 5000, 300_000)])
def test_sizes_at_the_edges(nb, np_, G):
    """Items of 4096 build and 16384 probe rows, chunks of 4096 groups; groups
    that leave a compact entry room and that do not."""
    _run_and_check([_instance(nb, np_, G, nb + G, gmin=-3)])


@pytest.mark.parametrize("values", [(-(1 << 20), 1 << 20), (-5, -1), (-(1 << 62), 1 << 62),
                                    (0, 1 << 41), (1 << 38, 1 << 39)])
@pytest.mark.parametrize("G", [5, 3000])
def test_value_ranges(values, G):
    _run_and_check([_instance(20_000, 120_000, G, 7, values)])


@pytest.mark.parametrize("skew", [3, 12, 60])
@pytest.mark.parametrize("G", [40, 20_000])
def test_skews(skew, G):
    _run_and_check([_instance(30_000, 300_000, G, skew, skew=skew)])


def _crowded(n=3000, m=9000):
    """Keys whose rotated hashes share their top 21 bits: one home bucket."""
    rng = np.random.default_rng(9)
    rot = (np.uint64(5) << np.uint64(43)) | rng.integers(0, 1 << 43, n, dtype=np.uint64)
    k = np.unique((rot >> np.uint64(21)) | (rot << np.uint64(43)))
    with np.errstate(over="ignore"):
        for c in (0xc4ceb9fe1a85ec53, 0xff51afd7ed558ccd):
            k ^= k >> np.uint64(33)
            k *= np.uint64(pow(c, -1, 1 << 64))
        k ^= k >> np.uint64(33)
    key = k.view(np.int64)
    return (key, rng.integers(0, 20, len(key)).astype(np.int32),
            key[rng.integers(0, len(key), m)], rng.integers(0, 1000, m), 0, 20)


@pytest.mark.parametrize("graph", [False, True])
def test_a_mix_of_instances_that_fail_their_first_pass(graph):
    hot = _instance(5_000, 200_000, 4000, 1)
    hot[1][:] = 17
    cases = [_instance(9_000, 50_000, 700, 2), _crowded(), hot,
             _instance(700, 9_000, 250_000, 3, (0, 1 << 50)),
             _instance(12_000, 60_000, 9_000, 4, (-(1 << 60), 1 << 60)),
             _instance(12_000, 60_000, 9_000, 5)]
    outside = _instance(3_000, 30_000, 100, 6)
    outside[1][::4] = 2000
    _run_and_check(cases + [outside], graph=graph)
