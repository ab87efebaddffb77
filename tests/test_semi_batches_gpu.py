"""The semi / anti join around a block's share of rows, every comparison, keys
that share a chain, the extreme keys and values, against numpy."""
import numpy as np
import pytest
import torch

from pageflow_b200 import tqpkernels
from tests.test_aggregate_gpu import _unmix64_array

pytestmark = pytest.mark.gpu
LOW = np.iinfo(np.int64).min
OPS = {1: np.not_equal, 2: np.less, 3: np.less_equal, 4: np.greater, 5: np.greater_equal}


def _expected(bk, bv, pk, pv, op, anti):
    vals = {}
    for k, v in zip(bk.tolist(), bv.tolist()):
        vals.setdefault(k, []).append(v)
    keep = [k in vals and (op == 0 or bool(OPS[op](np.array(vals[k]), v).any()))
            for k, v in zip(pk.tolist(), pv.tolist())]
    return np.nonzero(np.array(keep) != anti)[0]


@pytest.mark.parametrize("nb,np_", [(1, 1), (2, 7), (100, 4095), (5000, 4096), (5000, 4097),
                                    (20_011, 12_345)])
@pytest.mark.parametrize("op", range(6))
@pytest.mark.parametrize("anti", [False, True])
def test_batches(nb, np_, op, anti):
    rng = np.random.default_rng(nb + op)
    # half the keys from one chain: their hashes agree below the top nine bits
    chain = _unmix64_array(np.arange(40, dtype=np.uint64) << np.uint64(55) | np.uint64(77))
    pool = np.concatenate([chain, rng.integers(-1 << 60, 1 << 60, nb)])
    bk, pk = rng.choice(pool[:-1], nb), rng.choice(pool, np_)
    pk[rng.random(np_) < 0.1] = np.iinfo(np.int64).max
    bv, pv = rng.integers(-3, 4, nb), rng.integers(-3, 4, np_)
    bv[0], pv[0] = LOW, LOW
    host = torch.empty(2, dtype=torch.int64, pin_memory=True)
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (bk, pk, bv, pv)]
    rows = tqpkernels.join_semi_anti(t[0], t[1], t[2] if op else None, t[3] if op else None,
                                     op, anti, host)[:int(host[0])]
    assert int(host[1]) == 0
    assert np.array_equal(rows.cpu().numpy(), _expected(bk, bv, pk, pv, op, anti))
