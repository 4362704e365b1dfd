"""Sorts around the sizes where the kernel changes: one cluster up to 32768
pairs (1 to 8 CTAs of 1024 and more), tiles of 2048 below 393216, full tiles
above; with passes that move nothing and passes narrower than a digit."""
import numpy as np
import pytest
import torch

import oracle
from pimdal_b200 import _lib as L
from pimdal_b200 import ops

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 7, 33, 1023, 1024, 1025, 2049, 8191, 8193, 32767, 32768, 32769, 34817, 393215, 393216]


def stable(key, ids, dtype, begin, end):
    x = key.view(np.uint32) ^ (np.uint32(0x80000000) if dtype == L.I32 else np.uint32(0))
    d = (x >> np.uint32(begin)) & np.uint32((1 << (end - begin)) - 1)
    o = np.argsort(d, kind="stable")
    return key[o], ids[o]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("form", ["uniform", "few", "equal", "bits", "pairs", "keys"])
def test_short_sorts(ctx, n, form):
    rng = np.random.default_rng(n)
    key = rng.integers(-2**31, 2**31, n, dtype=np.int64).astype(np.int32)
    ids = rng.integers(-2**31, 2**31, n, dtype=np.int64).astype(np.int32)
    dtype = L.I32 if n % 2 else L.U32
    begin, end = 0, 32
    if form == "few":  # two middle passes move nothing
        key &= np.int32(0x0F0000FF)
    if form == "equal":
        key[:] = -5
    if form == "bits":
        begin, end = 3, 22
    kt, it = torch.from_numpy(key).cuda(), torch.from_numpy(ids).cuda()
    want_k, want_i = stable(key, ids, dtype, begin, end)
    if form == "pairs":
        pairs = torch.stack([kt, it], 1).contiguous().view(torch.int64).view(-1)
        out, _ = ops.sort_kernel(ctx, pairs, key_dtype=dtype, layout=L.LAYOUT_PAIRS)
        ctx.sync()
        got = out.view(torch.int32).view(n, 2).cpu().numpy()
        assert np.array_equal(got[:, 0], want_k) and np.array_equal(got[:, 1], want_i)
        return
    out, ptr = ops.sort_kernel(ctx, kt, it if form != "keys" else None, key_dtype=dtype, begin_bit=begin,
                               end_bit=end, want_ptr=form != "keys")
    ctx.sync()
    assert np.array_equal(out.cpu().numpy(), want_k)
    if form != "keys":
        assert np.array_equal(ptr.cpu().numpy(), want_i)
    if form == "uniform" and dtype == L.U32:
        ek, ep = oracle.sort_pairs(key.view(np.uint32))
        out, ptr = ops.sort_kernel(ctx, kt, key_dtype=dtype)
        ctx.sync()
        assert np.array_equal(out.cpu().numpy().view(np.uint32), ek)
        assert np.array_equal(ptr.cpu().numpy().view(np.uint32), ep)


def test_replayed_capture_sorts_new_data(ctx):
    n = 5000
    key = torch.randint(-2**31, 2**31 - 1, (n,), dtype=torch.int32, device="cuda")
    out, ptr = torch.empty_like(key), torch.empty_like(key)
    run = lambda: ops.sort_kernel(ctx, key, key_dtype=L.I32, out=out, out_ptr=ptr)
    run()
    ctx.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    for seed in range(3):
        key.copy_(torch.randint(-2**31, 2**31 - 1, (n,), dtype=torch.int32, device="cuda"))
        graph.replay()
        ctx.sync()
        want, order = torch.sort(key, stable=True)
        assert torch.equal(out, want) and torch.equal(ptr, order.to(torch.int32))
