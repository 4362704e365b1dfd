"""The fused scan's expressions against numpy in wrapping int64: expressions
that begin with the terms of the one before and ones that only look so, sums
beyond 32 bits and of both signs, in private and in shared table copies."""
import numpy as np
import pytest
import torch

from pimdal_b200 import _lib as L
from pimdal_b200 import ops

pytestmark = pytest.mark.gpu

N = 100_003


@pytest.mark.parametrize("keys", [1, 2, 6, 40, 1024])
def test_expressions(ctx, keys):
    rng = np.random.default_rng(keys)
    a = rng.integers(-2**40, 2**40, N)
    b = rng.integers(-100, 100, N).astype(np.int32)
    c = rng.integers(0, 256, N).astype(np.uint8)
    k = rng.integers(0, keys, N).astype(np.int32)
    d = rng.integers(-2**31, 2**31, N, dtype=np.int64).astype(np.int32)
    t = {n: torch.from_numpy(x).cuda() for n, x in dict(a=a, b=b, c=c, k=k, d=d).items()}
    A, B, Cc = a.astype(np.int64), b.astype(np.int64), c.astype(np.int64)
    sets = [
        # chains of one, two and three terms; then a chain broken by another column
        ([[t["a"]], [t["a"], (t["b"], 1, 100)], [t["a"], (t["b"], 1, 100), (t["c"], 0, 7)], [t["c"]],
          [t["b"], (t["c"], 0, 7)]],
         [A, A * (100 - B), A * (100 - B) * (Cc + 7), Cc, B * (Cc + 7)]),
        # the same column with another sign or addend, and as another type, is another term
        ([[(t["b"], 0, 1)], [(t["b"], 1, 1), t["a"]], [(t["b"], 0, 2), t["a"], t["a"]], [3], [3, t["a"]],
          [(t["b"], 0, 0, L.U32), t["c"]]],
         [B + 1, (1 - B) * A, (B + 2) * A * A, np.full(N, 3), 3 * A, (B & 0xFFFFFFFF) * Cc]),
    ]
    pred = [(t["d"], ops.make_pred(L.PRED_GE, -2**30))]
    take = d >= -2**30
    for exprs, want in sets:
        res, outs = ops.select_aggregate(ctx, N, preds=pred, group=[(t["k"], 1)] if keys > 1 else (),
                                         key_space=keys, exprs=exprs)
        ctx.sync()
        g = int(res.item())
        kk = (k if keys > 1 else np.zeros(N, np.int32))[take]
        cnt = np.bincount(kk, minlength=keys)
        have = np.nonzero(cnt)[0]
        assert g == have.size and np.array_equal(outs["key"][:g].cpu().numpy(), have)
        assert np.array_equal(outs["count"][:g].cpu().numpy(), cnt[have])
        for e, w in enumerate(want):
            sums = np.zeros(keys, np.int64)
            with np.errstate(over="ignore"):
                np.add.at(sums, kk, w[take])
            assert np.array_equal(outs[f"sum{e}"][:g].cpu().numpy(), sums[have]), e
