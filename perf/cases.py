"""Measured cases of the operator layer: what a database host has it do.

Each case is one call of a public operator on columns resident in HBM, with a
context, output columns and hash tables that the caller keeps between calls.
Sizes are those of this repository's configurations, tests and benchmark,
from one reference block (8000 rows) to 2^28 rows, with ragged ones between.
Output columns start zeroed, so the rows past a result's count compare equal.
"""
import functools
import math

import numpy as np
import torch

from pimdal_b200 import _lib as L
from pimdal_b200 import gen, ops, serve, tpch

DEV = "cuda:0"


def listed():
    return [
        # The reference's block size: a selection inside a short interactive
        # query, where the call itself costs more than its rows.
        {"name": "select_8k", "op": "select", "rows": 8000, "selectivity": 0.5, "dtype": "i32",
         "layout": "columns", "want_ptr": True},
        # The selection configuration: 2^24 int32 keys, one in ten kept.
        {"name": "select_16m", "op": "select", "rows": 1 << 24, "selectivity": 0.1, "dtype": "i32",
         "layout": "columns", "want_ptr": True},
        # A short ORDER BY or the sort of one index run: signed keys that
        # come with row ids of their own, a ragged count.
        {"name": "sort_100k", "op": "sort", "rows": 100_003, "dist": "zipf", "dtype": "i32",
         "layout": "columns", "given_ptr": True},
        # The sort configuration: 2^26 uniform (key, row id) pairs.
        {"name": "sort_64m", "op": "sort", "rows": 1 << 26, "dist": "uniform", "dtype": "u32",
         "layout": "columns", "given_ptr": False},
        # The sort-merge join configuration: R = 2^24, S = 2^26, both unsorted.
        {"name": "smj_16m_64m", "op": "smj", "inner": 1 << 24, "outer": 1 << 26},
        # A join with a small dimension: the table stays in L2.
        {"name": "hash_join_60k_1m", "op": "hash_join", "build": 60_001, "probe": 1_000_003,
         "dist": "uniform", "match_permille": 500},
        # The hash join configuration: 2^25 build rows, 2^28 probe rows, half
        # of which match.
        {"name": "hash_join_32m_256m", "op": "hash_join", "build": 1 << 25, "probe": 1 << 28,
         "dist": "uniform", "match_permille": 500},
        # GROUP BY over a mid-sized intermediate result: a ragged row count and
        # the configuration's middle group count.
        {"name": "group_10m_4k", "op": "group", "rows": 10_000_019, "groups": 1 << 12,
         "method": "hash", "dist": "uniform"},
        # The high-cardinality group-by configuration.
        {"name": "group_256m_4m", "op": "group", "rows": 1 << 28, "groups": 1 << 22,
         "method": "hash", "dist": "uniform"},
        # The sort method on skewed keys (the reference's second group-by).
        {"name": "group_sort_30m", "op": "group", "rows": 30_000_001, "groups": 100_000,
         "method": "sort", "dist": "zipf"},
        # TPC-H Q1's fused scan over a lineitem table of about 6e7 rows.
        {"name": "scan_q1_60m", "op": "scan", "orders": 15_000_000, "query": "q1"},
        # One served request: date filter, join with the orders table and
        # revenue by priority and flag, over half of the fact table.
        {"name": "served_30m", "op": "served", "orders": 15_000_000, "rows": 30_000_017,
         "date_share": 0.25, "dim": 0, "two_keys": True},
    ]


def _log(rng, lo, hi):
    """A whole number whose logarithm is uniform between those of lo and hi."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    op = rng.choice(["select", "sort", "smj", "hash_join", "group", "group", "scan", "served"])
    dtype = rng.choice(["i32", "u32"])
    layout = rng.choice(["columns", "columns", "pairs"])
    dist = rng.choice(["uniform", "uniform", "zipf"])
    if op == "select":
        return {"op": op, "rows": _log(rng, 1000, 1 << 28), "selectivity": round(rng.uniform(0.0, 1.0), 3),
                "dtype": dtype, "layout": layout, "want_ptr": rng.random() < 0.75}
    if op == "sort":
        return {"op": op, "rows": _log(rng, 1000, 1 << 26), "dist": dist, "dtype": dtype,
                "layout": layout, "given_ptr": rng.random() < 0.5}
    if op == "smj":
        outer = _log(rng, 4000, 1 << 26)
        return {"op": op, "inner": max(1, outer // rng.randint(1, 16)), "outer": outer}
    if op == "hash_join":
        probe = _log(rng, 8000, 1 << 28)
        return {"op": op, "build": max(1, min(1 << 25, probe // rng.randint(2, 64))), "probe": probe,
                "dist": dist, "match_permille": rng.choice([50, 500, 1000])}
    if op == "group":
        method = rng.choice(["hash", "hash", "sort"])
        rows = _log(rng, 8000, 1 << 28 if method == "hash" else 1 << 27)
        return {"op": op, "rows": rows, "groups": _log(rng, 4, min(rows, 1 << 22)), "method": method,
                "dist": dist}
    orders = _log(rng, 20_000, 15_000_000)
    if op == "scan":
        return {"op": op, "orders": orders, "query": rng.choice(["q1", "q6"])}
    return {"op": op, "orders": orders, "rows": _log(rng, orders // 2, 3 * orders),
            "date_share": round(rng.uniform(0.01, 0.5), 3), "dim": rng.randint(0, 1),
            "two_keys": rng.random() < 0.5}


@functools.lru_cache(maxsize=8)
def _zipf(n, s):
    return gen.zipf_cdf(n, s)


def _zeros(n, dtype=torch.int32):
    return torch.zeros(n, dtype=dtype, device=DEV)


def _keys(ctx, c, n, seed, dtype):
    """n keys over the whole 32-bit range: uniform, or Zipf(1.0) over 2^20 of them."""
    if c["dist"] == "zipf":
        return ops.gen_column(ctx, gen.Spec(L.GEN_PERM_ZIPF, dtype, seed=seed, cdf=_zipf(1 << 20, 1.0)), n)
    lo, hi = (0, 2**32 - 1) if dtype == L.U32 else (-2**31, 2**31 - 1)
    return ops.gen_column(ctx, gen.Spec(L.GEN_UNIFORM, dtype, seed=seed, lo=lo, hi=hi), n)


def _payload(ctx, n, seed, stream_id=1):
    return ops.gen_column(ctx, gen.Spec(L.GEN_UNIFORM, L.I32, seed=seed, stream_id=stream_id,
                                        lo=-2**31, hi=2**31 - 1), n)


def prepare(case, seed):
    c = case
    ctx = ops.Context(0)
    result = _zeros(1, torch.int64)
    dtype = L.U32 if c.get("dtype") == "u32" else L.I32
    pairs = c.get("layout") == "pairs"
    layout = L.LAYOUT_PAIRS if pairs else L.LAYOUT_COLUMNS
    if c["op"] == "select":
        n = c["rows"]
        keys = ops.gen_column(ctx, gen.Spec(L.GEN_UNIFORM, dtype, seed=seed, lo=0, hi=2**31 - 1), n)
        if pairs:
            keys = torch.stack([keys, torch.arange(n, dtype=torch.int32, device=DEV)], 1).view(torch.int64).view(-1)
        pred = ops.make_pred(L.PRED_LT, int(c["selectivity"] * 2**31))
        ptr = _zeros(n) if c["want_ptr"] and not pairs else None
        kw = dict(key_dtype=dtype, layout=layout, want_ptr=c["want_ptr"], out=torch.zeros_like(keys),
                  out_ptr=ptr, result=result)
        return lambda: ops.sel_kernel(ctx, keys, pred, **kw)
    if c["op"] == "sort":
        n = c["rows"]
        keys = _keys(ctx, c, n, seed, dtype)
        ptr = _payload(ctx, n, seed) if c["given_ptr"] and not pairs else None
        if pairs:
            keys = torch.stack([keys, torch.arange(n, dtype=torch.int32, device=DEV)], 1).view(torch.int64).view(-1)
        kw = dict(key_dtype=dtype, layout=layout, out=torch.zeros_like(keys),
                  out_ptr=None if pairs else _zeros(n))
        return lambda: ops.sort_kernel(ctx, keys, ptr, **kw)
    if c["op"] == "smj":
        ni, no = c["inner"], c["outer"]
        ik = ops.gen_column(ctx, gen.Spec(L.GEN_PERM, L.I32, seed=seed, perm_domain=ni), ni)
        ok = ops.gen_column(ctx, gen.Spec(L.GEN_PERM_UNIFORM, L.I32, seed=seed, stream_id=3, lo=0,
                                          hi=ni - 1, perm_domain=ni), no)
        ip, op = _payload(ctx, ni, seed), _payload(ctx, no, seed, 2)
        kw = dict(out_inner=_zeros(no), out_outer=_zeros(no), result=result, capacity=no)
        return lambda: ops.sort_merge_join(ctx, ik, ip, ok, op, **kw)
    if c["op"] == "hash_join":
        nb, npr = c["build"], c["probe"]
        cdf = _zipf(min(nb, 1 << 20), 0.75) if c["dist"] == "zipf" else None
        bk = ops.gen_column(ctx, gen.Spec(L.GEN_PERM, L.I32, seed=seed, perm_domain=2 * nb), nb)
        pk = ops.gen_column(ctx, gen.Spec(L.GEN_PROBE, L.I32, seed=seed, stream_id=2, lo=nb,
                                          perm_domain=2 * nb, match_permille=c["match_permille"],
                                          cdf=cdf), npr)
        bp = _payload(ctx, nb, seed)
        kw = dict(capacity=npr, out_payload=_zeros(npr), out_row=_zeros(npr), result=result)
        return lambda: ops.hash_join(ctx, bk, bp, pk, **kw)
    if c["op"] == "group":
        n, g = c["rows"], c["groups"]
        if c["dist"] == "zipf":
            spec = gen.Spec(L.GEN_PERM_ZIPF, L.I32, seed=seed, cdf=_zipf(min(g, 1 << 20), 1.0))
        else:
            spec = gen.Spec(L.GEN_PERM_UNIFORM, L.I32, seed=seed, stream_id=10, lo=0, hi=g - 1)
        keys = ops.gen_column(ctx, spec, n)
        vals = ops.gen_column(ctx, gen.Spec(L.GEN_UNIFORM, L.I64, seed=seed, stream_id=1, lo=100, hi=10**7), n)
        outs = {w: _zeros(2 * g, torch.int64) for w in ("sum", "count", "min", "max")}
        outs["key"] = _zeros(2 * g)
        method = L.GROUP_HASH if c["method"] == "hash" else L.GROUP_SORT
        kw = dict(method=method, expected_groups=g, capacity=2 * g, outs=outs, result=result)
        return lambda: ops.group_kernel(ctx, keys, vals, **kw)
    t = serve.Tables(ctx, orders=c["orders"], seed=seed)
    if c["op"] == "scan":
        li = tpch.Lineitem(ctx, t, seed=seed + 1)
        if c["query"] == "q6":
            preds, exprs = tpch.q6_args(li)
            group, space = (), 1
        else:
            pred, group, exprs = tpch.q1_args(li)
            preds, space = [pred], tpch.N_RFLAG * tpch.N_LSTATUS
        outs = {f"sum{e}": _zeros(space, torch.int64) for e in range(len(exprs))}
        outs |= {"key": _zeros(space), "count": _zeros(space, torch.int64)}
        kw = dict(preds=preds, group=group, key_space=space, exprs=exprs, outs=outs, result=result)
        return lambda: ops.select_aggregate(ctx, li.n, **kw)
    n = min(c["rows"], t.n)
    col, table, slots, flag, n_flag = t.dim(c["dim"])
    mult = n_flag if c["two_keys"] else 1
    space = t.n_attr(c["dim"]) * mult
    outs = {"key": _zeros(space), "sum": _zeros(space, torch.int64), "count": _zeros(space, torch.int64)}
    days = max(1, round(c["date_share"] * serve.DAYS))
    d0 = seed % (serve.DAYS - days + 1)
    kw = dict(flag=flag[:n] if c["two_keys"] else None, attr_mult=mult, key_space=space, outs=outs, result=result)
    args = (t.l_date[:n], d0, d0 + days - 1, col[:n], table, slots, t.l_price[:n], t.l_discount[:n])
    return lambda: ops.select_join_aggregate(ctx, *args, **kw)


def run(state):
    return state()


def work(case):
    """Bytes each case must read and write once; its arithmetic is integer and not counted."""
    c = case
    if c["op"] == "select":
        b = 8 if c["layout"] == "pairs" else 4
        per_kept = 8 if c["layout"] == "pairs" or c["want_ptr"] else 4
        return {"bytes": c["rows"] * (b + c["selectivity"] * per_kept)}
    if c["op"] == "sort":
        read = 8 if c["layout"] == "pairs" or c["given_ptr"] else 4
        return {"bytes": c["rows"] * (read + 8)}
    if c["op"] == "smj":  # every outer row matches one inner row
        return {"bytes": 8 * c["inner"] + 16 * c["outer"]}
    if c["op"] == "hash_join":
        return {"bytes": 8 * c["build"] + c["probe"] * (4 + 8 * c["match_permille"] / 1000)}
    if c["op"] == "group":
        return {"bytes": 12 * c["rows"] + 36 * c["groups"]}
    if c["op"] == "scan":
        n = 4 * c["orders"]  # 1 to 7 rows per order
        year, quantity, discount = 365 / 2557, 23 / 50, 3 / 11
        if c["query"] == "q6":
            return {"bytes": n * (4 + year * (4 + quantity * (4 + discount * 8)))}
        return {"bytes": n * (4 + 22 * 2436 / 2557)}
    n = min(c["rows"], 4 * c["orders"])
    return {"bytes": n * (4 + c["date_share"] * (16 + c["two_keys"]))}


def exact(case, seed):
    """Every output is a whole number or a copied value, so there is nothing to round."""
    return None
