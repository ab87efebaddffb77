"""The batch engine's values at the ends of int64, and a block's first rows of an
instance, whose groups' lanes of a warp are added together."""
import numpy as np
import pytest

from tests.test_batch_passes_gpu import _instance, _run_and_check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G", [7, 3000])
def test_values_at_the_ends_of_their_type(G):
    I = np.iinfo(np.int64)
    case = list(_instance(9_000, 70_000, G, 3))
    rng = np.random.default_rng(4)
    ends = np.array([I.min, I.min + 1, -1, 0, 1, I.max - 1, I.max, 1 << 39, -(1 << 39),
                     (1 << 62) + 5])
    case[3] = np.where(rng.random(70_000) < 0.01, rng.choice(ends, 70_000), case[3])
    _run_and_check([tuple(case)])
    case[3] = rng.choice(ends, 70_000)
    _run_and_check([tuple(case)])
