"""Operators whose tiles form look-back chains past one 4096-word block of
look-back words, with a ragged last tile, and chains of a batch that start
inside a block."""
import numpy as np
import pytest
import torch

import oracle
from pimdal_b200 import _lib as L
from pimdal_b200 import ops

pytestmark = pytest.mark.gpu


def rand(n, lo, hi, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(lo, hi, (n,), dtype=torch.int32, device="cuda", generator=g)


@pytest.mark.parametrize("tiles", [4095, 4096, 4097, 8193])
def test_merge_chain(ctx, tiles):
    n = 2048 * tiles - 5  # outer rows of a merge tile
    outer = torch.sort(rand(n, 0, 5000, tiles))[0]
    inner = torch.arange(0, 5000, 2, dtype=torch.int32, device="cuda")
    ids = torch.arange(n, dtype=torch.int32, device="cuda")
    res, oo, oi = ops.smj_merge(ctx, inner, inner * 3, outer, ids)
    ctx.sync()
    keep = outer % 2 == 0
    m = int(res.item())
    assert m == int(keep.sum())
    assert torch.equal(oo[:m], ids[keep]) and torch.equal(oi[:m], outer[keep] * 3)


@pytest.mark.parametrize("tiles", [4096, 8193])
def test_probe_chain(ctx, tiles):
    n = 3072 * tiles - 7  # rows of a probe tile
    probe = rand(n, 0, 3000, tiles)
    build = torch.arange(0, 3000, 3, dtype=torch.int32, device="cuda")
    res, pay, row = ops.hash_join(ctx, build, build + 7, probe, partition_bits=0xFFFFFFFF)
    ctx.sync()
    keep = torch.nonzero(probe % 3 == 0).view(-1).to(torch.int32)
    m = int(res.item())
    assert m == keep.numel()
    assert torch.equal(row[:m], keep) and torch.equal(pay[:m], probe[keep.long()] + 7)


def test_batch_chains_inside_blocks(ctx):
    sizes = [1, 3071, 3073, 700_001, 12_000_000, 5, 900_000]
    outs, wants, keep = [], [], []
    for i, n in enumerate(sizes):
        bk = torch.arange(0, 4000, 2, dtype=torch.int32, device="cuda")
        pk = rand(n, 0, 4000, 100 + i)
        op, orow = torch.empty_like(pk), torch.empty_like(pk)
        outs.append((op, orow))
        hit = torch.nonzero(pk % 2 == 0).view(-1)
        wants.append((pk[hit] + 1, hit.to(torch.int32)))
        keep.append((bk, bk + 1, pk))
    args = [ops.hash_join_args(k[0], k[1], k[2], None, o[0], o[1]) for k, o in zip(keep, outs)]
    batch = ops.Batch(ctx, L.BATCH_HASH_JOIN, args)
    for _ in range(2):
        batch.run()
        ctx.sync()
        for (pay, row), (op, orow), m in zip(wants, outs, batch.results.tolist()):
            assert m == pay.numel()
            assert torch.equal(op[:m], pay) and torch.equal(orow[:m], row)
    batch.close()


def test_small_selection_chain(ctx):
    n = (1 << 20) - 3  # 256 tiles of 4096 rows
    keys = np.random.default_rng(1).integers(-2**31, 2**31, n, dtype=np.int64).astype(np.int32)
    kt = torch.from_numpy(keys).cuda()
    for seed in range(3):
        res, out, ptr = ops.sel_kernel(ctx, kt, ops.make_pred(L.PRED_LT, seed * 10**9))
        ctx.sync()
        ov, op = oracle.select(keys, -2**63, seed * 10**9 - 1)
        m = int(res.item())
        assert m == ov.size and np.array_equal(out[:m].cpu().numpy(), ov)
        assert np.array_equal(ptr[:m].cpu().numpy().view(np.uint32), op)
