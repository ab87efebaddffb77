"""KeyedPass1 where the one-read route's memory does not fit: the general route
answers, as it did for every chunk before."""
import pytest
import torch

from pageflow_b200 import keyed_aggregate
from pageflow_b200.keyed_aggregate import KeyedPass1, _as_2d

pytestmark = pytest.mark.gpu

AGGS = [("sum", 1), ("count", None), ("avg", 1), ("min", 1), ("max", 1)]


def _chunk(n, groups):
    g = torch.Generator(device="cuda").manual_seed(n)
    key = torch.randperm(n, generator=g, device="cuda") % groups
    return {0: key * 11 + 3, 1: torch.randint(-500, 10_000, (n,), generator=g, device="cuda")}


# 2M rows of 700K groups take a second, larger table
@pytest.mark.parametrize("n,groups", [(2_000_000, 700_000), (900_000, 1000), (5_000, 70)])
@pytest.mark.parametrize("room", [0, 100 << 20])
@pytest.mark.parametrize("B", [1, 8])
def test_no_room_for_the_table(monkeypatch, n, groups, room, B):
    cols = _chunk(n, groups)
    p = KeyedPass1([0], AGGS)
    real, general, asked = keyed_aggregate._native.workspace, p._hash_and_sort, []

    def workspace(nbytes, device):
        asked.append(nbytes)
        if nbytes > room:
            raise torch.OutOfMemoryError("no room")
        return real(nbytes, device)

    def hash_and_sort(c, k):   # the general route has room
        monkeypatch.setattr(keyed_aggregate._native, "workspace", real)
        return general(c, k)

    monkeypatch.setattr(keyed_aggregate._native, "workspace", workspace)
    monkeypatch.setattr(p, "_hash_and_sort", hash_and_sort)
    out, buckets = p.pass1(cols, B)
    monkeypatch.setattr(keyed_aggregate._native, "workspace", real)
    assert len(asked) == (2 if room and n == 2_000_000 else 1)
    want = general(cols, [_as_2d(cols[0])])
    assert len(out) == len(want) and all(torch.equal(a, b) for a, b in zip(out, want))
    assert (buckets is None) == (B == 1)
    if B > 1:
        assert torch.equal(buckets[0], keyed_aggregate.hash_buckets(want[0], B)[0])
