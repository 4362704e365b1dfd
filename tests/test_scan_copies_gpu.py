"""The fused scan's copies of its sums, from one per thread down to one per CTA:
every sum against numpy, and the cost of adding the copies up."""
import numpy as np
import pytest
import torch

from pimdal_b200 import _lib as L
from pimdal_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exprs", [0, 1, 6])
@pytest.mark.parametrize("keys", [1, 2, 7, 8, 9, 33, 65, 300, 650, 700, 1024])
def test_against_numpy(ctx, keys, exprs):
    n = 70_001
    rng = np.random.default_rng(keys)
    a = rng.integers(-2**62, 2**62, n)
    b = rng.integers(-100, 100, n).astype(np.int32)
    k = rng.integers(0, keys, n).astype(np.int32)
    at, bt, kt = (torch.from_numpy(x).cuda() for x in (a, b, k))
    terms = [[at], [bt], [at, bt], [(bt, 1, 7)], [at, at], [bt, bt]][:exprs]
    res, outs = ops.select_aggregate(ctx, n, preds=[(bt, ops.make_pred(L.PRED_LT, 60))],
                                     group=[(kt, 1)] if keys > 1 else (), key_space=keys, exprs=terms)
    ctx.sync()
    sel = b < 60
    kk, a, b = k[sel] if keys > 1 else np.zeros(sel.sum(), np.int32), a[sel], b[sel].astype(np.int64)
    cnt = np.bincount(kk, minlength=keys)
    have = np.nonzero(cnt)[0]
    assert int(res.item()) == have.size and np.array_equal(outs["key"][: have.size].cpu().numpy(), have)
    assert np.array_equal(outs["count"][: have.size].cpu().numpy(), cnt[have])
    with np.errstate(over="ignore"):
        for e, w in enumerate([a, b, a * b, 7 - b, a * a, b * b][:exprs]):
            sums = np.zeros(keys, np.int64)
            np.add.at(sums, kk, w)
            assert np.array_equal(outs[f"sum{e}"][: have.size].cpu().numpy(), sums[have]), e


def test_cost_of_the_copies(ctx):
    """A count by 30 keys, 64 copies, took 1.6 times as long as by 6 keys when
    all lanes read one bank."""
    n = 3_000_000

    def ms(keys):
        key = torch.randint(0, keys, (n,), dtype=torch.int32, device="cuda")
        best = 1e9
        for _ in range(20):
            x, y = torch.cuda.Event(True), torch.cuda.Event(True)
            x.record()
            ops.select_aggregate(ctx, n, group=[(key, 1)], key_space=keys)
            y.record()
            y.synchronize()
            best = min(best, x.elapsed_time(y))
        ctx.sync()
        return best

    assert ms(30) < 1.35 * ms(6)
