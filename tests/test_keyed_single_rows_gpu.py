"""KeyedPass1 over chunks of single rows: after one that the one-read route gave
up on, the next seven of integer columns do not try it, and answer the same."""
import pytest
import torch

from pageflow_b200.keyed_aggregate import KeyedPass1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.int64, torch.float64])
def test_chunks_after_one_of_single_rows(dtype):
    n = 1_500_000
    g = torch.Generator(device="cuda").manual_seed(3)
    v = torch.randint(-9, 1 << 20, (n,), generator=g, device="cuda").to(dtype)
    single = {0: torch.randperm(n, generator=g, device="cuda"), 1: v}
    few = {0: single[0] % 1000, 1: v}
    p = KeyedPass1([0], [("sum", 1), ("count", None), ("avg", 1)])
    one_read, tried = p._one_read, []
    p._one_read = lambda *a: tried.append(1) or one_read(*a)
    want = KeyedPass1([0], p.aggs).pass1(few, 8)
    p.pass1(single, 8)
    for chunk in range(1, 10):
        out, buckets = p.pass1(few, 8)
        assert all(torch.equal(a, b) for a, b in zip(out, want[0]))   # whole sums, in floats too
        assert torch.equal(buckets[0], want[1][0]) and buckets[1] == want[1][1]
        assert len(tried) == (1 + max(0, chunk - 7) if dtype == torch.int64 else 1 + chunk)
