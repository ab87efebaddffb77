"""Null rows of gathered one-word columns: the null element repeated along the
row, at every word width and element size."""
import pytest
import torch

from pageflow_b200 import gather

pytestmark = pytest.mark.gpu

COLUMNS = [(torch.int8, ()), (torch.uint8, (2,)), (torch.int16, ()), (torch.uint8, (4,)),
           (torch.float16, (2,)), (torch.int32, ()), (torch.float32, ()), (torch.int16, (4,)),
           (torch.float32, (2,)), (torch.int64, ()), (torch.float64, ()), (torch.int8, (16,)),
           (torch.bfloat16, (8,)), (torch.int32, (4,)), (torch.float64, (2,)), (torch.int64, (2,))]


@pytest.mark.parametrize("n", [1, 3, 1023, 1025, 40_001])
@pytest.mark.parametrize("share", [0.0, 0.3, 1.0])
def test_null_rows_of_every_width(n, share):
    g = torch.Generator(device="cuda").manual_seed(n)
    rows = 777
    cols = [torch.randint(0, 100, (rows,) + s, generator=g, device="cuda").to(d) for d, s in COLUMNS]
    idx = torch.randint(0, rows, (n,), generator=g, device="cuda")
    null = torch.rand(n, generator=g, device="cuda") < share
    idx[null] = gather.NULL
    # together in one launch, and each by itself
    for got in (gather.index_with_null_many(cols, idx),
                [gather.index_with_null_many([c], idx)[0] for c in cols]):
        for out, col in zip(got, cols):
            want = col[idx.clamp_min(0)]
            want[null] = torch.full((1,), gather.NULL, dtype=col.dtype, device="cuda")
            assert torch.equal(out, want)
