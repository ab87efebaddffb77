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


def _rows_of_groups(order, nb, G, seed, values=(0, 1 << 24)):
    """An instance whose probe rows' groups are `order`."""
    rng = np.random.default_rng(seed)
    key = rng.permutation(np.unique(rng.integers(-(1 << 62), 1 << 62, nb + 9)))[:nb]
    grp = (np.arange(nb) % G).astype(np.int32)
    fk = key[order + G * rng.integers(0, nb // G, len(order))]
    return key, grp, fk, rng.integers(*values, len(order)), 0, G


# lanes of a group in a warp: none alike, pairs, fours, all, and a few hot ones
@pytest.mark.parametrize("lanes", ["apart", "2", "3", "4", "7", "32", "hot"])
@pytest.mark.parametrize("values", [(0, 1 << 24), (-(1 << 20), 1 << 20), (-(1 << 60), 1 << 60)])
def test_groups_of_a_warps_lanes(lanes, values):
    G, n = 6000, 300_007
    rng = np.random.default_rng(len(lanes))
    if lanes == "apart":
        order = np.arange(n) % G
    elif lanes == "hot":
        order = np.where(rng.random(n) < 0.7, 11, rng.integers(0, G, n))
    else:
        order = (np.arange(n) // int(lanes) * 17) % G
    case = _rows_of_groups(order, 12_000, G, 5, values)
    misses = case[2].copy()
    misses[rng.random(n) < 0.2] = 1 << 62   # lanes without a group between them
    _run_and_check([case, (case[0], case[1], misses, *case[3:])])


@pytest.mark.parametrize("n", [1, 31, 255, 256, 511, 513])
def test_fewer_rows_than_a_first_step(n):
    _run_and_check([_rows_of_groups(np.arange(n) // 5 % 700, 1400, 700, n)])
