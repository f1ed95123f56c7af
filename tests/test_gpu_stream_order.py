"""A call sees inputs that the program has queued on the default stream just before it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_inputs_still_being_written_on_the_default_stream(cuda):
    import torch
    from openmeeg_gb300 import api, workloads
    w = workloads.small(1)
    geo = api.Geometry.from_head(w.head)
    ref = api.DipSourceMat(geo, w.dipoles).cpu().numpy()
    src = torch.as_tensor(w.dipoles, device=cuda).contiguous()
    d = torch.zeros_like(src)
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)   # some 50 ms of waiting on the default stream, then the dipoles arrive
    d.copy_(src)
    assert np.array_equal(api.DipSourceMat(geo, d).cpu().numpy(), ref)
