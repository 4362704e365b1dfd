"""High-cardinality hash group-by around 2^25 rows, where 65537 to 131072
expected groups take one partition pass of 6 bits and whole-SM chunk tables
instead of two passes and half tables: against the sort method on the device,
and the count and sum of all rows."""
import pytest
import torch

from pimdal_b200 import _lib as L
from pimdal_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2**25 - 1, 2**25 + 3])
@pytest.mark.parametrize("groups", [66_560, 100_000, 131_072])
@pytest.mark.parametrize("offset", [0, 1])
def test_against_the_sort_method(ctx, groups, n, offset):
    g = torch.Generator(device="cuda").manual_seed(groups + n)
    ids = torch.randperm(2**22, dtype=torch.int32, device="cuda", generator=g)[:groups] * 977
    ids[0] = -1  # the all-ones key takes the global table
    pick = torch.randint(0, groups, (n + offset,), device="cuda", generator=g)
    keys = ids[pick][offset:]
    vals = torch.randint(-2**62, 2**62, (n + offset,), device="cuda", generator=g)[offset:]
    got = {}
    for method in (L.GROUP_HASH, L.GROUP_SORT):
        res, outs = ops.group_kernel(ctx, keys, vals, method=method, expected_groups=groups,
                                     capacity=groups)
        ctx.sync()
        assert int(res.item()) == groups  # 250 rows of each on average
        got[method] = outs
    for name in ("key", "sum", "count", "min", "max"):
        assert torch.equal(got[L.GROUP_HASH][name], got[L.GROUP_SORT][name]), name
    assert torch.equal(got[L.GROUP_HASH]["key"], ids.sort().values)
    assert int(got[L.GROUP_HASH]["count"].sum()) == n
    assert int(got[L.GROUP_HASH]["sum"].sum()) == int(vals.sum())  # mod 2^64
