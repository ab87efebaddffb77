"""The first tick of a run: its columns' rows are as many as its keys, as an
assignment to the buffers' first rows asks."""
import pytest
import torch

from pageflow_b200.sorted_run_merge import merge_sorted_unique_runs_inplace

pytestmark = pytest.mark.gpu


def _buffers(device, n=100):
    return (torch.zeros(n, dtype=torch.int64, device=device),
            [torch.zeros(n, dtype=torch.int64, device=device),
             torch.zeros((n, 2), dtype=torch.float64, device=device)])


@pytest.mark.parametrize("device", ["cuda", "cpu"])
@pytest.mark.parametrize("rows", [11, 9, 0, 100])
@pytest.mark.parametrize("column", [0, 1])
def test_a_column_of_other_rows_is_refused(device, rows, column):
    key, bufs = _buffers(device)
    tick = torch.arange(10, device=device)
    vals = [torch.ones(10, dtype=torch.int64, device=device),
            torch.ones((10, 2), dtype=torch.float64, device=device)]
    vals[column] = torch.ones((rows,) + vals[column].shape[1:], dtype=vals[column].dtype,
                              device=device)
    with pytest.raises(RuntimeError):
        merge_sorted_unique_runs_inplace(key, bufs, 0, tick, vals, ["sum", "sum"])


@pytest.mark.parametrize("device", ["cuda", "cpu"])
def test_what_an_assignment_takes(device):
    """One row or a number for all of them, other types, and buffers in strides."""
    key, bufs = _buffers(device)
    tick = torch.arange(10, device=device)
    for vals, want in (([torch.tensor([7], device=device), torch.full((1, 2), 3.0, device=device)],
                        (7, 3.0)),
                       ([torch.tensor(5, device=device), torch.tensor(2.5, device=device)],
                        (5, 2.5)),
                       ([torch.full((10,), 4, dtype=torch.int32, device=device),
                         torch.full((10, 2), 1.5, dtype=torch.float32, device=device)], (4, 1.5))):
        assert merge_sorted_unique_runs_inplace(key, bufs, 0, tick, vals, ["sum", "sum"]) == 10
        assert torch.equal(key[:10], tick) and bool((bufs[0][:10] == want[0]).all())
        assert bool((bufs[1][:10] == want[1]).all()) and not bufs[1][10:].any()
    wide = torch.zeros((100, 4), dtype=torch.float64, device=device)
    vals = [torch.full((10,), 6, dtype=torch.int64, device=device),
            torch.arange(20, dtype=torch.float64, device=device).view(10, 2)]
    merge_sorted_unique_runs_inplace(key, [bufs[0], wide[:, 1:3]], 0, tick, vals, ["sum", "sum"])
    assert torch.equal(wide[:10, 1:3], vals[1]) and not wide[:, 0].any() and not wide[10:].any()
