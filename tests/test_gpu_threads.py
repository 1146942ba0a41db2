"""Solves of different sizes enqueued by two host threads at once. A kernel's limit of dynamic shared memory belongs to the
function, which all threads and streams of a context share: a call that lowered it to its own need would make another
thread's launch of the same build fail. Both threads enqueue on one stream, so that only their host code runs at once."""

import ctypes
import threading

import pytest
import torch

from mit_jax_b200 import capi
from mit_jax_b200 import cg2d as cg
from mit_jax_b200.synthetic import make_batch

pytestmark = pytest.mark.gpu


def _args(N, count, tile, **kw):
    """One prepared cg2d_solve_groups call (one iteration) and everything it points to."""
    syn, B = make_batch(N, 1, tile)
    dev = torch.device("cuda")
    ex = cg.default_exchanger(syn.L)
    b = torch.as_tensor(B["b"]).to(dev).expand(count, *B["b"].shape[1:]).contiguous()
    ops = [torch.as_tensor(B[k]).to(dev).expand_as(b).contiguous() for k in cg.OPS]
    x0, x, dg = torch.zeros_like(b), torch.empty_like(b), torch.zeros((count, capi.DIAG_BYTES), dtype=torch.uint8, device=dev)
    params = capi.default_params()
    for k, v in kw.items():
        setattr(params, k, v)
    arr = (capi.Group * 1)()
    g = arr[0]
    g.topo, g.count, g.nrhs, g.cg2dNorm = ex.handle(dev), count, 1, float(B["cg2dNorm"][0])
    for name, t in zip(cg.OPS, ops):
        setattr(g, name, t.data_ptr())
    g.b[0], g.x0[0], g.x_out[0], g.diag[0], g.tolerance[0], g.max_iters[0] = (
        b.data_ptr(), x0.data_ptr(), x.data_ptr(), dg.data_ptr(), 0.0, 1)
    nbytes = capi.lib().cg2d_workspace_size(arr, 1, ctypes.byref(params))
    assert nbytes > 0
    ws = torch.empty(nbytes + 256, dtype=torch.uint8, device=dev)
    base = ws.data_ptr() + (-ws.data_ptr()) % 256
    return (arr, 1, ctypes.byref(params), base, nbytes), (ex, b, ops, x0, x, dg, ws, params)


@pytest.mark.parametrize("case", ["on_chip", "streamed"])
def test_two_threads_with_different_shared_memory(case):
    if case == "on_chip":      # 36 and 171 KB a CTA of the same team build
        calls = [_args(90, 1, None), _args(90, 16, None)]
    else:                      # the streaming kernel at two pipeline depths (grid_ctas too small for the state)
        calls = [_args(90, 1, None, grid_ctas=8, ctas_per_sm=1, stages=s) for s in (2, 4)]
    stream = torch.cuda.current_stream().cuda_stream
    L = capi.lib()
    for args, _ in calls:
        assert L.cg2d_solve_groups(*args, stream) == capi.CG2D_OK
    torch.cuda.synchronize()
    bad, go = [], threading.Barrier(2)

    def work(args):
        go.wait()
        for n in range(1500):
            st = L.cg2d_solve_groups(*args, stream)
            if st != capi.CG2D_OK:
                bad.append((n, st))
                return

    threads = [threading.Thread(target=work, args=(args,)) for args, _ in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert bad == []
