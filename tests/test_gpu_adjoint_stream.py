"""Gain and gradients on a stream that the context is not bound to, while earlier work on that stream is still queued:
the same as on the default stream, and the context's own binding is left as it was."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bound", [False, True])
def test_gradients_on_a_side_stream(cuda, bound):
    import torch
    from openmeeg_gb300 import adjoint, api, workloads
    w = workloads.small(1, layers=3)
    ctx = api.Context(0)
    geo = api.Geometry.from_meshes(w.head.vertices, w.head.triangles, w.head.domains, ctx=ctx)
    sig0 = torch.tensor([d[2] for d in w.head.domains], dtype=torch.float64)
    dip0 = torch.as_tensor(w.dipoles[:5], dtype=torch.float64, device=cuda)
    bar = torch.randn(len(w.electrodes) + len(w.squids), 5, dtype=torch.float64, device=cuda,
                      generator=torch.Generator(device=cuda).manual_seed(1))

    def grads(wait):
        sig, dip = sig0.clone().requires_grad_(True), (dip0 * 1.0).requires_grad_(True)
        wait()
        G = adjoint.gain(sig, dip + 0.0, geo, w.head.domains, w.electrodes, w.squids)
        wait()
        return [G.detach(), *torch.autograd.grad((G * bar).sum(), [sig, dip])]

    want = [x.cpu() for x in grads(lambda: None)]
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    if bound:
        with torch.cuda.stream(a):
            ctx.bind_current_stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(b):
        got = [x.cpu() for x in grads(lambda: torch.cuda._sleep(50_000_000))]
    for x, y in zip(got, want):
        assert torch.equal(x, y)
    assert ctx.stream == (a.cuda_stream if bound else 0)
