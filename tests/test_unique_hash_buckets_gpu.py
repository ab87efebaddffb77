"""The unique hash's bucket table: chains of full buckets whose slots share a
fingerprint, both ways to size the table, one and two keys, against numpy."""
import numpy as np
import pytest
import torch

from pageflow_b200 import tqpkernels
from tests.test_aggregate_gpu import _unmix64_array

pytestmark = pytest.mark.gpu


def _join(build, probe):
    host = torch.empty(2, dtype=torch.int64, pin_memory=True)
    b, p = tqpkernels.join_unique_hash([torch.from_numpy(x).cuda() for x in build],
                                       [torch.from_numpy(x).cuda() for x in probe], host)
    n = int(host[0])
    return b[:n].cpu().numpy(), p[:n].cpu().numpy()


def _expected(build, probe):
    rows = {k: i for i, k in enumerate(zip(*[x.tolist() for x in build]))}
    hit = [(rows[k], j) for j, k in enumerate(zip(*[x.tolist() for x in probe])) if k in rows]
    return (np.array([h[0] for h in hit], np.int64), np.array([h[1] for h in hit], np.int64))


@pytest.mark.parametrize("chain", [7, 8, 9, 17, 300, 511])
def test_one_bucket_and_fingerprint(chain):
    """Keys whose hashes differ in their top nine bits alone, which neither the
    home bucket nor the fingerprint sees, one of them left out of the build."""
    low = np.uint64(0x0012_3456_789A_BCDE)
    keys = _unmix64_array(np.arange(chain + 1, dtype=np.uint64) << np.uint64(55) | low)
    rng = np.random.default_rng(chain)
    other = rng.integers(-1 << 40, 1 << 40, 2000)
    build = [np.unique(np.concatenate([keys[:-1], other[:1000]]))]
    build[0] = build[0][rng.permutation(len(build[0]))]
    probe = [np.concatenate([keys, other, keys])]
    for got, want in zip(_join(build, probe), _expected(build, probe)):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("nb,np_", [(1, 1), (2, 3), (3, 5000), (2049, 4097), (100_003, 300_007)])
@pytest.mark.parametrize("two", [False, True])
def test_sizes(nb, np_, two):
    rng = np.random.default_rng(nb)
    build = [rng.permutation(2 * nb)[:nb].astype(np.int64) - nb // 2]
    probe = [rng.integers(-nb, 2 * nb, np_)]
    if two:
        build = [build[0] >> 2, (build[0] & 3) - 2]
        probe = [probe[0] >> 2, (probe[0] & 3) - 2]
    for got, want in zip(_join(build, probe), _expected(build, probe)):
        assert np.array_equal(got, want)


# 0.3 full up to 5,033,164 build rows, where the probe side has the room for it
@pytest.mark.parametrize("nb,np_", [(5_033_164, 8_400_000), (5_033_165, 8_400_000),
                                    (100_000, 166_666), (100_000, 166_672), (6_000_001, 400_009)])
def test_both_loads(nb, np_):
    rng = np.random.default_rng(3)
    keys = rng.permutation(nb).astype(np.int64)
    fk = rng.integers(-5, nb + 5, np_)
    inv = np.empty(nb, np.int64)
    inv[keys] = np.arange(nb)
    b, p = _join([keys], [fk])
    hit = np.nonzero((fk >= 0) & (fk < nb))[0]
    assert np.array_equal(p, hit)
    assert np.array_equal(b, inv[fk[hit]])


def test_probe_rows_written_over_the_probe_keys():
    """The row output may be the probe key column itself, as the rows are
    written after the last key is read."""
    from pageflow_b200 import _native as N
    L = N.lib()
    rng = np.random.default_rng(4)
    build, probe = rng.permutation(5000).astype(np.int64), rng.integers(0, 9000, 40_000)
    b, p = torch.from_numpy(build).cuda(), torch.from_numpy(probe).cuda()
    host = torch.empty(2, dtype=torch.int64, pin_memory=True)
    bi = torch.empty(40_000, dtype=torch.int64, device="cuda")
    ws = N.workspace(L.pf_join_unique_hash_workspace(5000, 40_000), b.device)
    N.check(L.pf_join_unique_hash(b.data_ptr(), None, 5000, p.data_ptr(), None, 40_000, 1,
                                  bi.data_ptr(), p.data_ptr(), host.data_ptr(), ws.data_ptr(),
                                  ws.numel(), N.stream_of(b.device)), "join")
    n = int(host[0])
    for got, want in zip((bi[:n].cpu().numpy(), p[:n].cpu().numpy()),
                         _expected([build], [probe])):
        assert np.array_equal(got, want)
