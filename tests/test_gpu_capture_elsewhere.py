"""A call on the library's own stream while the program captures a blocking stream of its own: the call works and the
capture goes on.  In relaxed mode by the calling thread, in thread-local mode by another one."""
import ctypes
import glob
import threading

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,other_thread", [(2, False), (2, True), (1, True)])
def test_call_beside_a_capture(cuda, mode, other_thread):
    import torch
    from openmeeg_gb300 import api, workloads
    libs = glob.glob("/usr/local/cuda/lib64/libcudart.so*")
    if not libs:
        pytest.skip("no shared CUDA runtime to capture with")
    rt = ctypes.CDLL(libs[0])
    w = workloads.small(1)
    geo = api.Geometry.from_head(w.head)
    d = torch.as_tensor(w.dipoles, device=cuda)
    ref = api.DipSourceMat(geo, d).clone()   # (the second output's memory is torch's already)
    api.DipSourceMat(geo, d)
    torch.cuda.synchronize()
    s, g = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(s)) == 0
    begun, done, codes = threading.Event(), threading.Event(), []

    def capture():
        rt.cudaSetDevice(0)
        codes.append(rt.cudaStreamBeginCapture(s, mode))
        begun.set()
        done.wait(60)
        codes.append(rt.cudaStreamEndCapture(s, ctypes.byref(g)))

    t = None
    if other_thread:
        t = threading.Thread(target=capture)
        t.start()
        begun.wait(60)
    else:
        codes.append(rt.cudaStreamBeginCapture(s, mode))
    try:
        out = api.DipSourceMat(geo, d)
    finally:
        if t is None:
            codes.append(rt.cudaStreamEndCapture(s, ctypes.byref(g)))
        else:
            done.set()
            t.join()
        rt.cudaStreamDestroy(s)
    assert codes == [0, 0]
    assert torch.equal(out, ref)
