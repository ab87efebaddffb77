"""The host wait's limit (pf_set_wait_timeout_ms): any number of milliseconds."""
import pytest
import torch

from pageflow_b200 import _native
from pageflow_b200.join_aggregate import JoinAggregate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ms", [60_000, 1 << 40, (1 << 63) // 1000 + 1, (1 << 63) - 1])
def test_a_large_limit_ends_no_wait(ms):
    L = _native.lib()
    n = 6_000_000   # milliseconds of work: the first poll finds it unfinished
    key = torch.arange(n, dtype=torch.int64, device="cuda")
    plan = JoinAggregate(n, n, 0, 10, "cuda", autotune=False)
    L.pf_set_wait_timeout_ms(ms)
    try:
        for _ in range(3):
            keys, sums, counts = plan.run(key, (key % 10).to(torch.int32), key, key)
    finally:
        L.pf_set_wait_timeout_ms(120_000)   # the default
    assert counts.tolist() == [n // 10] * 10
    assert sums.tolist() == [int(key[i::10].sum()) for i in range(10)]
