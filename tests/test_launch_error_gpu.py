"""A launch that the runtime refuses is reported by the call that made it and
by no later one."""
import ctypes as C
import types

import pytest
import torch

from pimdal_b200 import _lib as L
from pimdal_b200 import ops

pytestmark = pytest.mark.gpu

RELAXED = 2  # cudaStreamCaptureModeRelaxed


@pytest.fixture
def refusing_stream():
    """A stream whose capture has been broken: launches on it are refused by the host."""
    torch.cuda.synchronize()
    rt = C.CDLL("libcudart.so.12")
    s, graph = C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreateWithFlags(C.byref(s), 1) == 0
    assert rt.cudaStreamBeginCapture(s, RELAXED) == 0
    assert rt.cudaStreamSynchronize(s) != 0  # not allowed while capturing: ends the capture
    rt.cudaGetLastError()
    yield rt, types.SimpleNamespace(cuda_stream=s.value)
    rt.cudaGetLastError()
    rt.cudaStreamEndCapture(s, C.byref(graph))
    rt.cudaGetLastError()
    rt.cudaStreamDestroy(s)


def test_next_call_succeeds(ctx, refusing_stream):
    rt, bad = refusing_stream
    n = 1000
    g = torch.Generator(device="cuda").manual_seed(1)
    bk = torch.randperm(n, device="cuda", generator=g).int()
    pk = torch.randint(0, 2 * n, (n,), dtype=torch.int32, device="cuda", generator=g)
    d = torch.zeros(n, dtype=torch.int32, device="cuda")
    v = torch.ones(n, dtype=torch.int64, device="cuda")
    table = ops.hash_kernel(ctx, bk, bk, table_size=4096)
    runs = [lambda **kw: ops.hash_join(ctx, bk, bk, pk, **kw)[0],
            lambda **kw: ops.hj_probe(ctx, table, 4096, pk, **kw)[0],
            lambda **kw: ops.sort_kernel(ctx, pk, **kw)[0],
            lambda **kw: ops.group_kernel(ctx, pk, v, expected_groups=2 * n, **kw)[0],
            lambda **kw: ops.select_aggregate(ctx, n, exprs=[[v]], **kw)[0],
            lambda **kw: ops.select_join_aggregate(ctx, d, 0, 1, pk, table, 4096, v, d, key_space=n, **kw)[0]]
    for run in runs:
        run()  # workspaces
    ctx.sync()
    for run in runs:
        want = run().clone()
        with pytest.raises(L.PimdalError) as e:
            run(stream=bad)
        assert e.value.status == 6  # PIMDAL_ERR_CUDA
        assert rt.cudaPeekAtLastError() == 0
        assert torch.equal(run(), want)
        ctx.sync()
