"""The domain of a dipole just off a surface is that of the FP64 solid angles.

At a distance h from a triangle of edge a, FP32 cannot tell the sign of the
triangle's solid angle from h / a of about 1e-7 down, and the FP64 formula drops
it where 4 A h < 2e-10.  Heads of three sizes and two densities; points off faces,
edges and corners, on both sides of every interface.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _off_surface(head, rng, n):
    out = []
    for V, T in zip(head.vertices, head.triangles):
        V, T = np.asarray(V), np.asarray(T)
        p = V[T[rng.integers(0, len(T), n)]]
        b = rng.dirichlet([1, 1, 1], n)
        b[n // 2:3 * n // 4] = [0.5, 0.5, 0.0]
        b[3 * n // 4:] = [1.0, 0.0, 0.0]
        x = np.einsum("nk,nkc->nc", b, p)
        nn = np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
        nn /= np.linalg.norm(nn, axis=1, keepdims=True)
        h = 10.0 ** rng.uniform(-12, -3, n) * rng.choice([-1, 1], n) * np.abs(V).max()
        out.append(x + h[:, None] * nn)
    x = np.vstack(out)
    return np.hstack([x, rng.standard_normal(x.shape)])


@pytest.mark.parametrize("subdiv,scale", [(1, 1.0), (2, 1.0), (2, 0.1), (1, 1e-4), (2, 1e13)])
def test_domains_just_off_a_surface(cuda, subdiv, scale):
    import torch
    from openmeeg_gb300 import _lib, api, synthetic as syn
    head = syn.nested_head(subdiv, [0.6 * scale, 0.8 * scale, scale], [1.0, 0.0125, 1.0], perturb_seed=4, perturb_amp=0.05)
    geo = api.Geometry.from_head(head)
    dip = torch.as_tensor(_off_surface(head, np.random.default_rng(subdiv), 240), device=cuda)
    dom = torch.full((len(dip),), -7, dtype=torch.int32, device=cuda)
    _lib.check(geo.lib.omg_dipole_domains_dev(geo.ctx.handle, geo.handle, ctypes.c_void_p(dip.data_ptr()), len(dip),
                                              ctypes.c_void_p(dom.data_ptr())))   # by FP64 sums
    dom = dom.cpu().numpy()
    dip, dom = dip[torch.as_tensor(dom >= 0, device=cuda)].contiguous(), dom[dom >= 0]   # (-1: sums that contradict each other)
    assert len(dom) > 360
    it = _lib.Integrator(3, 0, 1e-3)
    got = api.DipSourceMat(geo, dip, it).T.cpu().numpy()
    for d in sorted(set(dom)):
        sel = np.nonzero(dom == d)[0]
        want = api.DipSourceMat(geo, dip[torch.as_tensor(sel, device=cuda)], it, geo.domain_names[d]).T.cpu().numpy()
        assert np.array_equal(got[sel], want, equal_nan=True)
    conducting = np.array([head.domains[d][2] != 0.0 for d in dom])
    assert api.Surf2VolMat(geo, dip[:, :3]).shape[0] == conducting.sum()
