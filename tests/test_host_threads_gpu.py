"""Two host threads, each with a context and a stream of its own, run the fused
passes at the same time with tables of different sizes: every call is launched
and its result is right."""
import ctypes as C
import threading

import pytest
import torch

from pimdal_b200 import _lib as L
from pimdal_b200 import ops

pytestmark = pytest.mark.gpu

CALLS = 4000


def column(n, lo, hi, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(lo, hi, (n,), dtype=dtype, device="cuda", generator=g)


def run_threads(calls):
    """calls: per thread a function returning a status; all run CALLS times side by side."""
    bad, start = [], threading.Barrier(len(calls))

    def work(i, call):
        start.wait()
        bad.extend((i, st) for st in (call() for _ in range(CALLS)) if st)

    threads = [threading.Thread(target=work, args=ic) for ic in enumerate(calls)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    return bad


@pytest.mark.parametrize("spaces", [(15, 50), (256, 4096)])
def test_join_pass(spaces):
    n = 1000
    calls, checks, keep = [], [], []
    for i, ks in enumerate(spaces):
        c, stream = ops.Context(0), torch.cuda.Stream()
        keys = torch.arange(ks, dtype=torch.int32, device="cuda")
        table = ops.hash_kernel(c, keys, keys, table_size=16384)
        date, jkey = column(n, 0, 10, torch.int32, i), column(n, 0, ks, torch.int32, 10 + i)
        price, disc = column(n, -2**40, 2**40, torch.int64, 20 + i), column(n, 0, 100, torch.int32, 30 + i)
        outs = {"key": torch.zeros(ks, dtype=torch.int32, device="cuda")}
        outs |= {w: torch.zeros(ks, dtype=torch.int64, device="cuda") for w in ("sum", "count")}
        res = torch.zeros(1, dtype=torch.int64, device="cuda")
        c.reserve(16 * ks)
        a = L.SelectJoinAggregateArguments(
            size=n, date=date.data_ptr(), date_lo=0, date_hi=4, jkey=jkey.data_ptr(),
            table_ptr=table.data_ptr(), table_size=16384, price=price.data_ptr(),
            discount=disc.data_ptr(), attr_mult=1, key_space=ks, out_key=outs["key"].data_ptr(),
            out_sum=outs["sum"].data_ptr(), out_count=outs["count"].data_ptr(), out_capacity=ks)
        calls.append(lambda c=c, a=a, res=res, s=stream: c.lib.pimdal_select_join_aggregate(
            c.handle, C.byref(a), res.data_ptr(), s.cuda_stream))
        keep.append((keys, table, date, jkey, price, disc, a))
        take = date <= 4
        cnt = torch.bincount(jkey[take], minlength=ks)
        sums = torch.zeros(ks, dtype=torch.int64, device="cuda")
        sums.index_add_(0, jkey[take], price[take] * (100 - disc[take]))
        checks.append((c, stream, res, outs, cnt, sums))
    torch.cuda.synchronize()
    assert run_threads(calls) == []
    for c, stream, res, outs, cnt, sums in checks:
        c.sync(stream)
        have = cnt.nonzero().flatten()
        g = int(res.item())
        assert g == have.numel() and torch.equal(outs["key"][:g].long(), have)
        assert torch.equal(outs["count"][:g], cnt[have]) and torch.equal(outs["sum"][:g], sums[have])
        c.close()


@pytest.mark.parametrize("spaces", [(1, 1024), (40, 1000)])
def test_scan(spaces):
    n = 1000
    calls, checks, keep = [], [], []
    for i, ks in enumerate(spaces):
        c, stream = ops.Context(0), torch.cuda.Stream()
        key = column(n, 0, ks, torch.int32, i)
        val = [column(n, -2**40, 2**40, torch.int64, 10 * i + e) for e in range(6)]
        a = L.SelectAggregateArguments(size=n, n_preds=0, n_group=1, key_space=ks, n_exprs=6)
        a.group[0] = L.GroupCol(col=key.data_ptr(), dtype=L.I32, mult=1)
        outs = [torch.zeros(ks, dtype=torch.int64, device="cuda") for _ in range(7)]
        out_key = torch.zeros(ks, dtype=torch.int32, device="cuda")
        res = torch.zeros(1, dtype=torch.int64, device="cuda")
        for e in range(6):
            a.expr[e] = ops._expr([val[e]])
            a.out_sum[e] = outs[e].data_ptr()
        a.out_key, a.out_count, a.out_capacity = out_key.data_ptr(), outs[6].data_ptr(), ks
        c.reserve(8 * ks * 7)
        calls.append(lambda c=c, a=a, res=res, s=stream: c.lib.pimdal_select_aggregate(
            c.handle, C.byref(a), res.data_ptr(), s.cuda_stream))
        keep.append((key, val, a))
        want = [torch.zeros(ks, dtype=torch.int64, device="cuda").index_add_(0, key, v) for v in val]
        checks.append((c, stream, res, out_key, outs, want + [torch.bincount(key, minlength=ks)]))
    torch.cuda.synchronize()
    assert run_threads(calls) == []
    for c, stream, res, out_key, outs, want in checks:
        c.sync(stream)
        have = want[6].nonzero().flatten()
        g = int(res.item())
        assert g == have.numel() and torch.equal(out_key[:g].long(), have)
        for got, w in zip(outs, want):
            assert torch.equal(got[:g], w[have])
        c.close()
