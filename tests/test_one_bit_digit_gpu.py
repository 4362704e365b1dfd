"""A digit of one bit anywhere in the key: the bits above it do not move a row,
and nothing is written past the end of the outputs."""
import numpy as np
import pytest
import torch

import oracle
from pimdal_b200 import _lib as L
from pimdal_b200 import ops

pytestmark = pytest.mark.gpu

GUARD = 4096


def guarded(n):
    t = torch.full((n + GUARD,), 0x5A5A5A5A, dtype=torch.int32, device="cuda")
    return t, t[:n]


def check(full, n, want):
    got = full.cpu().numpy()
    assert np.array_equal(got[:n].view(np.uint32), want)
    assert np.all(got[n:] == 0x5A5A5A5A)


@pytest.mark.parametrize("n", [1, 32768, 32769, 400_003])
@pytest.mark.parametrize("bit", [0, 1, 12, 30, 31])
def test_sort(ctx, n, bit):
    keys = np.random.default_rng(n + bit).integers(0, 2**32, n, dtype=np.uint32)
    kt = torch.from_numpy(keys.view(np.int32)).cuda()
    for dtype, flip in ((L.U32, 0), (L.I32, 0x80000000)):
        order = np.argsort(((keys ^ np.uint32(flip)) >> np.uint32(bit)) & np.uint32(1), kind="stable")
        for want_ptr in (True, False):
            (of, out), (pf, ptr) = guarded(n), guarded(n)
            ops.sort_kernel(ctx, kt, key_dtype=dtype, begin_bit=bit, end_bit=bit + 1, out=out,
                            out_ptr=ptr if want_ptr else None, want_ptr=want_ptr)
            ctx.sync()
            check(of, n, keys[order])
            if want_ptr:
                check(pf, n, order.astype(np.uint32))


@pytest.mark.parametrize("n", [1, 5121, 100_003])
@pytest.mark.parametrize("shift", [1, 9, 31, 32])
def test_two_partitions(ctx, n, shift):
    keys = np.random.default_rng(n + shift).integers(0, 2**32, n, dtype=np.uint32)
    (of, out), (pf, ptr) = guarded(n), guarded(n)
    _, _, sizes = ops.part_kernel(ctx, torch.from_numpy(keys.view(np.int32)).cuda(), shift=shift, part_n=2,
                                  out=out, out_ptr=ptr)
    ctx.sync()
    ok, op, es = oracle.part_hash0(keys, shift=shift, part_n=2)
    check(of, n, ok)
    check(pf, n, op)
    assert np.array_equal(sizes.cpu().numpy(), es.astype(np.int64))
