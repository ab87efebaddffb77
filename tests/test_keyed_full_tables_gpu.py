"""KeyedPass1's table at its fullest, two thirds: chunks whose every row is a
group of its own, and second tables, are answered without the general route."""
import pytest
import torch

from pageflow_b200.keyed_aggregate import KeyedPass1

pytestmark = pytest.mark.gpu


def _pass1(key, v, aggs, B=1):
    p = KeyedPass1([0], aggs)

    def no_general_route(columns, keys):
        raise AssertionError("the table gave up")
    p._hash_and_sort = no_general_route
    return p.pass1({0: key, 1: v}, B)[0]


# 3 n / 2 places up to a power of two: the last rows before it and one past, to the
# largest first table of eight words a group
@pytest.mark.parametrize("n", [682, 683, 10_922, 10_923, 20_000, 21_845, 174_762, 300_000,
                               349_525])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_a_table_at_its_fullest(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    key = torch.randperm(n, generator=g, device="cuda") * (2 * seed + 1) + seed
    v = torch.randint(-100, 1 << 40, (n,), generator=g, device="cuda")
    out = _pass1(key, v, [("sum", 1), ("min", 1), ("max", 1), ("avg", 1)], 8 if seed else 1)
    order = torch.argsort(out[1])
    by_key = v[torch.argsort(key)]
    assert torch.equal(out[1][order], torch.sort(key)[0])
    assert torch.equal(out[2][order], by_key) and torch.equal(out[3][order], by_key)
    assert torch.equal(out[4][order], by_key.clamp_min(0))
    assert bool((out[0][1:] > out[0][:-1]).all())


# one table holds 699,050 groups of four words; more of them take a second
@pytest.mark.parametrize("groups", [340_000, 520_000, 640_000, 690_000, 720_000, 850_000, 1_000_000])
def test_groups_around_the_largest_first_table(groups):
    n = 4_000_000
    g = torch.Generator(device="cuda").manual_seed(groups)
    key = torch.randint(0, groups, (n,), generator=g, device="cuda")
    v = torch.randint(-100, 1 << 40, (n,), generator=g, device="cuda")
    out = _pass1(key, v, [("sum", 1), ("min", 1), ("max", 1), ("count", None)])
    k = out[1]
    s = torch.zeros(groups, dtype=torch.int64, device="cuda").index_add_(0, key, v)
    c = torch.bincount(key, minlength=groups)
    assert k.numel() == int((c > 0).sum())
    assert torch.equal(out[2], s[k]) and torch.equal(out[5], c[k])
