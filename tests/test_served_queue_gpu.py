"""The fused date filter -> join -> group-by pass at the edges of its 128-row
steps and of the queue of selected rows: ragged sizes, an unaligned date column,
none, some and all rows selected, keys that find no, one or several build rows,
per-warp and per-CTA tables, sums of both signs beyond 32 bits."""
import numpy as np
import pytest
import torch

from pimdal_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 4097, 300_007])
@pytest.mark.parametrize("share,attrs,dup", [(0.0, 5, 1), (0.02, 5, 1), (0.3, 200, 3), (1.0, 1000, 1)])
def test_against_numpy(ctx, n, offset, share, attrs, dup):
    rng = np.random.default_rng(n + attrs)
    m = n + offset
    date = rng.integers(0, 1000, m).astype(np.int32)
    jkey = rng.integers(0, 4000, m).astype(np.int32)
    jkey[::97] = -1  # all ones: build rows of that key and an all-ones attribute are kept aside
    price = rng.integers(-2**40, 2**40, m)
    disc = rng.integers(0, 101, m).astype(np.int32)
    flag = rng.integers(0, 3, m).astype(np.uint8)
    bkey = np.concatenate([np.arange(0, 4000, 2)] * dup + [[-1]]).astype(np.int32)
    battr = rng.integers(0, attrs, bkey.size).astype(np.int32)
    cu = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    size = 16384
    table = ops.hash_kernel(ctx, cu(bkey), cu(battr), table_size=size)
    col = lambda x: cu(x)[offset:]
    hi = int(1000 * share) - 1
    res, outs = ops.select_join_aggregate(ctx, col(date), 0, hi, col(jkey), table, size, col(price),
                                          col(disc), flag=col(flag), attr_mult=3, key_space=3 * attrs)
    ctx.sync()
    sums, cnt = np.zeros(3 * attrs, np.int64), np.zeros(3 * attrs, np.int64)
    by_key = {}
    for k, a in zip(bkey.tolist(), battr.tolist()):
        by_key.setdefault(k, []).append(a)
    rows = np.nonzero(date[offset:] <= hi)[0] + offset
    for r in rows.tolist():
        for a in by_key.get(int(jkey[r]), ()):
            g = a * 3 + int(flag[r])
            sums[g] += price[r] * (100 - int(disc[r]))
            cnt[g] += 1
    have = np.nonzero(cnt)[0]
    g = int(res.item())
    assert g == have.size
    assert np.array_equal(outs["key"][:g].cpu().numpy(), have)
    assert np.array_equal(outs["count"][:g].cpu().numpy(), cnt[have])
    assert np.array_equal(outs["sum"][:g].cpu().numpy(), sums[have])
