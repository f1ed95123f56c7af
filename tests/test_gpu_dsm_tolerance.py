"""Tolerances at which nothing is settled by the first level: negative (every node refined to the last level, as the
reference's comparison has it) and zero; and the derivatives at a negative one.  Against the oracle at the 1e-12 of the
other adaptive tests; finite differences as there."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("levels,tol", [(1, -1.0), (2, -1.0), (3, -1e-3), (2, 0.0), (3, 1e-15)])
def test_values(cuda, order, levels, tol):
    from openmeeg_gb300 import _lib, api, workloads
    from oracle import oracle
    w = workloads.small(1, layers=3, perturb=True)
    dip = np.asarray(w.dipoles[:3])
    D = api.DipSourceMat(api.Geometry.from_head(w.head), dip, integrator=_lib.Integrator(order, levels, tol)).cpu().numpy()
    want = oracle.dsm(oracle.digest(w.head), dip, order, levels, tol)
    assert rel(D, want) < 1e-12
    if order == 0 and tol < 0:   # three points: the first level alone is visibly another value
        assert rel(D, oracle.dsm(oracle.digest(w.head), dip, order, 0, 1e-3)) > 1e-9


def test_derivatives(cuda):
    import torch
    from openmeeg_gb300 import _lib, adjoint, api, workloads
    w = workloads.small(1, layers=3, perturb=True)
    geo = api.Geometry.from_head(w.head)
    sig = torch.tensor([d[2] for d in w.head.domains], dtype=torch.float64)
    dip0 = torch.as_tensor(w.dipoles[:2], dtype=torch.float64, device=cuda)
    bar = torch.randn(len(w.electrodes), 2, generator=torch.Generator().manual_seed(3), dtype=torch.float64).to(cuda)

    def loss(dip):
        return (adjoint.gain(sig, dip, geo, w.head.domains, w.electrodes, None,
                             dsm_integrator=_lib.Integrator(0, 2, -1.0)) * bar).sum()

    dip = dip0.clone().requires_grad_(True)
    (g,) = torch.autograd.grad(loss(dip), [dip])
    fd = np.zeros((2, 6))
    for j in range(2):
        for c in range(6):
            d = torch.zeros_like(dip0)
            d[j, c] = 1e-5
            fd[j, c] = (float(loss(dip0 + d)) - float(loss(dip0 - d))) / 2e-5
    assert rel(g.cpu().numpy(), fd) < 1e-7   # (truncation 1e-10 over distances of 0.1 and more, rounding 1e-15 / 1e-5)
