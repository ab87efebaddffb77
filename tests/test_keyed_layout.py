"""KeyedPass1's kept layout when two threads with columns of different types
share the object: a thread uses the one it looked up or made."""
import torch

from pageflow_b200.keyed_aggregate import KeyedPass1

AGGS = [("sum", 1), ("max", 1)]


def _columns(dtype):
    return [torch.zeros((4, 1), dtype=torch.int64)], {1: torch.zeros(4, dtype=dtype)}


class _Shared(KeyedPass1):
    """Every look at _laid finds what another thread has just put there."""

    @property
    def _laid(self):
        return self.others

    @_laid.setter
    def _laid(self, mine):
        pass


def test_another_threads_layout_is_not_taken():
    plain = KeyedPass1([0], AGGS)
    of = {d: plain._layout_of(*_columns(d)) for d in (torch.int64, torch.int32)}
    assert of[torch.int64][2] != of[torch.int32][2]   # MAX's output is of another type
    shared = _Shared.__new__(_Shared)
    shared.others = None
    KeyedPass1.__init__(shared, [0], AGGS)
    for mine, theirs in ((torch.int64, torch.int32), (torch.int32, torch.int64)):
        plain._laid = None
        plain._layout_of(*_columns(theirs))
        shared.others = plain._laid
        got = shared._layout_of(*_columns(mine))
        assert got[2] == of[mine][2] and got[4] == of[mine][4]


def test_the_layout_is_kept_for_the_same_types():
    p = KeyedPass1([0], AGGS)
    assert p._layout_of(*_columns(torch.int64)) is p._layout_of(*_columns(torch.int64))
    assert p._layout_of(*_columns(torch.float64)) is None   # a float's maximum
