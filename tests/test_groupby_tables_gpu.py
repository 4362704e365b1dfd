"""The hash group-by's shared-memory tables at the edges of their modes: one
accumulator per lane up to 128 expected groups, one table per CTA up to 4608,
partitioned chunks above; groups beyond the expected count leave the shared
tables; sums carry between their two 32-bit words; unaligned columns."""
import numpy as np
import pytest
import torch

import oracle
from pimdal_b200 import _lib as L
from pimdal_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("groups,expected", [(1, 1), (128, 128), (129, 129), (212, 128), (4608, 4608),
                                             (4609, 4609), (6785, 128), (9000, 4608)])
def test_table_modes_and_carries(ctx, groups, expected, offset):
    n = 200_003
    rng = np.random.default_rng(groups * 3 + offset)
    keys = rng.integers(-2**31, 2**31, groups, dtype=np.int64).astype(np.int32)
    keys[0] = -1  # the all-ones key takes the global table
    k = keys[rng.integers(0, groups, n + offset)]
    # both signs, low words near 2^32, and a spread over all 64 bits
    v = np.where(rng.random(n + offset) < 0.5, rng.integers(-2**33, 2**33, n + offset),
                 rng.integers(-2**62, 2**62, n + offset))
    v[::3] = 2**32 - 1
    kt, vt = torch.from_numpy(k).cuda()[offset:], torch.from_numpy(v).cuda()[offset:]
    res, outs = ops.group_kernel(ctx, kt, vt, method=L.GROUP_HASH, expected_groups=expected,
                                 capacity=groups + 1)
    try:
        ctx.sync()
    except L.PimdalError as e:  # the global table is sized by the hint: too small is reported
        assert groups > 2048 and groups > 2 * expected and e.status == 4
        return
    g = int(res.item())
    exp = oracle.group_by(k[offset:], v[offset:])
    for name, want in zip(("key", "sum", "count", "min", "max"), exp):
        assert np.array_equal(outs[name][:g].cpu().numpy(), want), name


@pytest.mark.parametrize("groups", [65536, 65537, 100_000, 131_072, 131_073, 300_000])
def test_partition_counts(ctx, groups):
    """Around the group count where one partition pass becomes two, and the
    chunk tables that go with it."""
    n = 1_500_001
    rng = np.random.default_rng(groups)
    keys = rng.permutation(2**22)[:groups].astype(np.int32) * 977
    k = keys[rng.integers(0, groups, n)]
    v = rng.integers(-2**40, 2**40, n)
    res, outs = ops.group_kernel(ctx, torch.from_numpy(k).cuda(), torch.from_numpy(v).cuda(),
                                 method=L.GROUP_HASH, expected_groups=groups, capacity=groups)
    ctx.sync()
    g = int(res.item())
    for name, want in zip(("key", "sum", "count", "min", "max"), oracle.group_by(k, v)):
        assert np.array_equal(outs[name][:g].cpu().numpy(), want), name
