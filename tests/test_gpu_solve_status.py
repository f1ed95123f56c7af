"""A solve reports what its kernels reported on the device.

A wait that gives up leaves OMG_ERR_TIMEOUT in the context's status word and the
right-hand sides half updated.  No wait is made to give up here: a copy on another
stream writes the status while a solve of some tens of milliseconds runs.
"""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_solve_reports_a_status_of_its_kernels(cuda, precision):
    import torch
    from openmeeg_gb300 import _lib, api, workloads
    ctx = api.Context(0)
    w = workloads.config0(1)
    geo = api.Geometry.from_meshes(w.head.vertices, w.head.triangles, w.head.domains, ctx=ctx)
    sv = api.Solver(geo, precision=precision)
    hook = ctx.lib.omg_internal_status_dev
    hook.restype, hook.argtypes = ctypes.c_void_p, [ctypes.c_void_p]
    status = torch.as_tensor(api._DevView(hook(ctx.handle), (1,)), device=cuda).view(torch.int32)
    n = 30000
    B = torch.randn(geo.size, n, dtype=torch.float64, device=cuda)
    ref = sv.solve(B[:, :8])
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    code = torch.full((1,), -8, dtype=torch.int32, device=cuda)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(16_000_000)   # about 8 ms: the solve has begun and is not over
        status[:1].copy_(code, non_blocking=True)
    with pytest.raises(_lib.OMGError) as e:
        sv.solve(B)
    assert e.value.code == -8
    torch.cuda.synchronize()
    assert torch.equal(sv.solve(B[:, :8]), ref)   # the next call starts from a clear status
