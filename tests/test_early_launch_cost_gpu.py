"""Kernels that are launched early leave the SMs to run as they would behind an
ordinary launch: joins behind partition passes, merges behind sorts."""
import pytest
import torch

from pimdal_b200 import ops

pytestmark = pytest.mark.gpu


def ms(ctx, run):
    best = 1e9
    for _ in range(6):
        a, b = torch.cuda.Event(True), torch.cuda.Event(True)
        a.record()
        run()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    ctx.sync()
    return best


def test_hash_join_of_64_partitions(ctx):
    """1.5 times the time of 16 partitions when the clear was launched early."""
    nb, n = 8_000_000, 1 << 24
    build = torch.randperm(2 * nb, dtype=torch.int32, device="cuda")[:nb]
    probe = torch.randint(0, 2 * nb, (n,), dtype=torch.int32, device="cuda")
    pay, row = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))

    def join(bits):
        return ms(ctx, lambda: ops.hash_join(ctx, build, build, probe, partition_bits=bits, out_payload=pay,
                                             out_row=row))

    assert join(6) < 1.2 * join(4)


def test_merge_of_repeated_keys(ctx):
    """Each key 8 times on both sides: 2.3 times the time of unique inner keys when
    the merge came onto the SMs during the sorts."""
    n = 300_000
    inner = torch.randperm(n, dtype=torch.int32, device="cuda")
    outer = torch.randint(0, n, (n,), dtype=torch.int32, device="cuda")
    out = [torch.empty(9 * n, dtype=torch.int32, device="cuda") for _ in range(2)]

    def join(times):
        a, b = inner // times, outer // times
        return ms(ctx, lambda: ops.sort_merge_join(ctx, a, inner, b, outer, capacity=9 * n, out_inner=out[0],
                                                   out_outer=out[1]))

    assert join(8) < 1.6 * join(1)
