"""The adaptive dipole integrals: pairs that the first level does not settle are
integrated by a warp each, and the derivatives follow the same tree.

Dipoles down to 1 % of the head's radius from the innermost interface, every
rule, depths from none to the stack's limit, and numbers of listed pairs that
are no multiple of a CTA's warps.  A value is a sum over the same tree as the
oracle's; at a distance of 0.01 the subtraction r - r0 costs two digits and the
powers up to |x|^-5 a factor 5, so 5e-14 of rounding per term against 1e-12.
Tolerance 0 lists every pair, a huge one none: neither has a decision that a
finite difference could cross.  Its truncation is (1e-6 / 0.01)^2 x 30 < 1e-6.
"""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


def _near(w, n):
    V, T = np.asarray(w.head.vertices[0]), np.asarray(w.head.triangles[0])
    rng = np.random.default_rng(5)
    c = V.mean(0)
    t = T[rng.integers(0, len(T), n)]
    b = rng.dirichlet([1, 1, 1], n)
    p = np.einsum("nk,nkc->nc", b, V[t]) - c
    r = np.linalg.norm(p, axis=1, keepdims=True)
    d = np.resize([0.01, 0.03, 0.1, 0.4], n)[:, None] * r.mean()
    q = rng.standard_normal((n, 3))
    return np.hstack([c + p * (r - d) / r, q])


@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("levels,tol,n", [(0, 1e-3, 3), (1, 1e-3, 1), (2, 0.0, 2), (10, 1e-3, 7), (10, 1e-6, 1)])
def test_values_match_the_oracle(cuda, order, levels, tol, n):
    from openmeeg_gb300 import _lib, api, workloads
    from oracle import oracle
    w = workloads.small(1, layers=3, perturb=True)
    dip = _near(w, n)
    geo = api.Geometry.from_head(w.head)
    D = api.DipSourceMat(geo, dip, integrator=_lib.Integrator(order, levels, tol)).cpu().numpy()
    assert rel(D, oracle.dsm(oracle.digest(w.head), dip, order, levels, tol)) < 1e-12


@pytest.mark.parametrize("order,levels,tol", [(3, 10, 1e9), (3, 0, 1e-3), (1, 3, 0.0), (3, 2, 0.0), (0, 1, 0.0)])
def test_derivatives_match_central_differences(cuda, order, levels, tol):
    import torch
    from openmeeg_gb300 import _lib, adjoint, api, workloads
    w = workloads.small(1, layers=3, perturb=True)
    geo = api.Geometry.from_head(w.head)
    sig = torch.tensor([d[2] for d in w.head.domains], dtype=torch.float64)
    dip0 = torch.as_tensor(_near(w, 3), dtype=torch.float64, device=cuda)
    bar = torch.randn(len(w.electrodes), 3, generator=torch.Generator().manual_seed(3), dtype=torch.float64).to(cuda)

    def loss(dip):
        G = adjoint.gain(sig, dip, geo, w.head.domains, w.electrodes, None,
                         dsm_integrator=_lib.Integrator(order, levels, tol))
        return (G * bar).sum()

    dip = dip0.clone().requires_grad_(True)
    (g,) = torch.autograd.grad(loss(dip), [dip])
    fd = np.zeros((3, 6))
    for j in range(3):
        for c in range(6):
            d = torch.zeros_like(dip0)
            d[j, c] = 1e-6
            fd[j, c] = (float(loss(dip0 + d)) - float(loss(dip0 - d))) / 2e-6
    assert rel(g.cpu().numpy(), fd) < 1e-5
