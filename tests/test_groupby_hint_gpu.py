"""Hash group-by whose expected group count is too low for the lane
accumulators: the rows after the overflow go to the CTA table, every row is
counted once, and the call costs no multiple of one with the right estimate.
An estimate too low for the global table is reported."""
import numpy as np
import pytest
import torch

import oracle
from pimdal_b200 import _lib as L
from pimdal_b200 import ops

pytestmark = pytest.mark.gpu


def rows(n, groups, order, seed):
    rng = np.random.default_rng(seed)
    keys = rng.permutation(np.arange(-5, groups - 5).astype(np.int32) * 977)
    keys[0] = -1  # the all-ones key takes the global table
    g = rng.integers(0, groups, n)
    if order == "sorted":  # most warps see few groups
        g.sort()
    if order == "late":  # the groups that overflow the table come in the last rows only
        g[: n - n // 10] %= 40
    return keys[g], rng.integers(-2**62, 2**62, n)


def check(outs, res, k, v):
    g = int(res)
    for name, want in zip(("key", "sum", "count", "min", "max"), oracle.group_by(k, v)):
        assert g == len(want) and np.array_equal(outs[name][:g].cpu().numpy(), want), name


@pytest.mark.parametrize("order", ["random", "sorted", "late"])
@pytest.mark.parametrize("groups,expected", [(100, 60), (160, 64), (213, 64), (300, 50), (1500, 64), (1500, 128),
                                             (2000, 1)])
@pytest.mark.parametrize("offset", [0, 1])
def test_overflow(ctx, groups, expected, order, offset):
    n = 2_000_003  # several steps of every warp
    k, v = rows(n + offset, groups, order, groups)
    kt, vt = torch.from_numpy(k).cuda()[offset:], torch.from_numpy(v).cuda()[offset:]
    res, outs = ops.group_kernel(ctx, kt, vt, method=L.GROUP_HASH, expected_groups=expected,
                                 capacity=groups)
    ctx.sync()
    check(outs, res, k[offset:], v[offset:])


@pytest.mark.parametrize("n", [700, 130_003])
def test_batch(ctx, n):
    inst, args = [], []
    # a batch sizes each global table by its estimate (at least 256 slots)
    for i, (groups, expected) in enumerate([(240, 64), (9, 9), (250, 5), (120, 120), (180, 50), (700, 700)]):
        k, v = rows(n, groups, ("random", "sorted", "late")[i % 3], i)
        kt, vt = torch.from_numpy(k).cuda(), torch.from_numpy(v).cuda()
        outs = {w: torch.empty(groups, dtype=torch.int64, device="cuda") for w in ("sum", "count", "min", "max")}
        outs["key"] = torch.empty(groups, dtype=torch.int32, device="cuda")
        args.append(ops.group_args(kt, vt, outs, expected_groups=expected))
        inst.append((k, v, kt, vt, outs))
    b = ops.Batch(ctx, L.BATCH_GROUP, args)
    for _ in range(2):
        b.run()
        ctx.sync()
        for i, (k, v, _, _, outs) in enumerate(inst):
            check(outs, b.results[i].item(), k, v)
    b.close()


def test_too_small_global_table(ctx):
    k, v = rows(200_003, 6785, "random", 1)
    ops.group_kernel(ctx, torch.from_numpy(k).cuda(), torch.from_numpy(v).cuda(), method=L.GROUP_HASH,
                     expected_groups=128, capacity=6785)
    with pytest.raises(L.PimdalError) as e:
        ctx.sync()
    assert e.value.status == 4  # PIMDAL_ERR_TABLE_FULL


@pytest.mark.parametrize("groups,expected", [(300, 64), (300, 100), (1000, 128)])
def test_cost_of_a_low_estimate(ctx, groups, expected):
    """10 to 20 times the cost of the right estimate when every row of an
    overflowing group went to the global table."""
    n = 1 << 24
    k = torch.randint(0, groups, (n,), dtype=torch.int32, device="cuda") * 977
    v = torch.randint(0, 2**40, (n,), dtype=torch.int64, device="cuda")

    def ms(hint):
        best = 1e9
        for _ in range(5):
            a, b = torch.cuda.Event(True), torch.cuda.Event(True)
            a.record()
            ops.group_kernel(ctx, k, v, method=L.GROUP_HASH, expected_groups=hint, capacity=groups)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        ctx.sync()
        return best

    assert ms(expected) < 3 * ms(groups)
