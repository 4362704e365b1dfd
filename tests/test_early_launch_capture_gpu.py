"""Operators whose kernels are launched early, captured into a CUDA graph and
replayed on new data."""
import pytest
import torch

from pimdal_b200 import _lib as L
from pimdal_b200 import ops

pytestmark = pytest.mark.gpu


def column(n, lo, hi, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(lo, hi, (n,), dtype=dtype, device="cuda", generator=g)


@pytest.mark.parametrize("n,groups,method", [(5000, 7, L.GROUP_HASH), (200_000, 1000, L.GROUP_HASH),
                                             (200_000, 9000, L.GROUP_HASH), (50_000, 300, L.GROUP_SORT),
                                             (500_000, 300, L.GROUP_SORT)])
def test_group_by(ctx, n, groups, method):
    keys = column(n, 0, groups, torch.int32, 1)
    vals = column(n, -2**40, 2**40, torch.int64, 2)
    outs = {w: torch.zeros(2 * groups, dtype=torch.int64, device="cuda") for w in ("sum", "count", "min", "max")}
    outs["key"] = torch.zeros(2 * groups, dtype=torch.int32, device="cuda")
    res = torch.zeros(1, dtype=torch.int64, device="cuda")
    run = lambda: ops.group_kernel(ctx, keys, vals, method=method, expected_groups=groups,
                                   capacity=2 * groups, outs=outs, result=res)
    run()
    ctx.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    for seed in range(3):
        keys.copy_(column(n, 0, groups, torch.int32, 10 + seed))
        vals.copy_(column(n, -2**40, 2**40, torch.int64, 20 + seed))
        graph.replay()
        ctx.sync()
        want_k, inv, cnt = torch.unique(keys, return_inverse=True, return_counts=True)
        g = int(res.item())
        sums = torch.zeros(want_k.numel(), dtype=torch.int64, device="cuda").index_add_(0, inv, vals)
        assert g == want_k.numel() and torch.equal(outs["key"][:g], want_k)
        assert torch.equal(outs["count"][:g], cnt) and torch.equal(outs["sum"][:g], sums)


def test_fused_scan(ctx):
    n = 100_001
    a, b = column(n, 0, 1000, torch.int32, 3), column(n, -2**40, 2**40, torch.int64, 4)
    outs = {k: torch.zeros(1, dtype=torch.int64, device="cuda") for k in ("count", "sum0")}
    outs["key"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    res = torch.zeros(1, dtype=torch.int64, device="cuda")
    run = lambda: ops.select_aggregate(ctx, n, preds=[(a, ops.make_pred(L.PRED_LT, 500))], exprs=[[b]],
                                       outs=outs, result=res)
    run()
    ctx.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    for seed in range(3):
        a.copy_(column(n, 0, 1000, torch.int32, 30 + seed))
        graph.replay()
        ctx.sync()
        assert int(outs["count"]) == int((a < 500).sum()) and int(outs["sum0"]) == int(b[a < 500].sum())
