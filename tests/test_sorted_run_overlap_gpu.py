"""Merges whose tick is a view of the run's own buffers: the values before the
merge are the ones combined."""
import pytest
import torch

from pageflow_b200.sorted_run_merge import merge_sorted_unique_runs_inplace

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [5, 300, 200_001])
@pytest.mark.parametrize("shift", [0, 1, 2])
def test_a_tick_of_the_runs_own_rows(R, shift):
    g = torch.Generator(device="cuda").manual_seed(R)
    key = torch.arange(R, device="cuda") * 3
    col = torch.randint(0, 1 << 40, (R,), generator=g, device="cuda")
    other = torch.randint(0, 1 << 40, (R,), generator=g, device="cuda")
    was, other_was = col.clone(), other.clone()
    # the tick: the keys from row `shift` on, with the values `shift` rows before theirs,
    # and for the other column this one's
    n = R - shift
    m = merge_sorted_unique_runs_inplace(key, [col, other], R, key[shift:].clone(),
                                         [col[:n], was[:n]], ["sum", "sum"])
    assert m == R
    assert torch.equal(col[shift:], was[shift:] + was[:n]) and torch.equal(col[:shift], was[:shift])
    assert torch.equal(other[shift:], other_was[shift:] + was[:n])


def test_columns_of_one_buffer_are_merged_in_place_or_not():
    """Two columns side by side, and one column passed twice."""
    both = torch.arange(2000, device="cuda").view(2, 1000).clone()
    was = both.clone()
    key = torch.arange(1000, device="cuda")
    ones = torch.ones(1000, dtype=torch.int64, device="cuda")
    merge_sorted_unique_runs_inplace(key, [both[0], both[1]], 1000, key.clone(), [ones, ones],
                                     ["sum", "sum"])
    assert torch.equal(both, was + 1)
    merge_sorted_unique_runs_inplace(key, [both[0], both[0]], 1000, key.clone(), [ones, ones],
                                     ["sum", "sum"])
    assert torch.equal(both[0], was[0] + 2) and torch.equal(both[1], was[1] + 1)
