"""The lookup of domains where an interface is made of three or six open meshes (sectors of the innermost sphere): each
subtends a part of the solid angle, which counts in the sum.  Mixed precision and the lookup of points against FP64 and the sphere."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[3, 6])
def geo(cuda, tmp_path_factory, request):
    n = request.param
    from openmeeg_gb300 import api, io, synthetic as syn
    d = tmp_path_factory.mktemp("sectors")
    V, T = syn.icosphere(2)
    phi = np.arctan2(*V[T].mean(1)[:, 1::-1].T)
    sector = np.clip(((phi + np.pi) * n / (2 * np.pi)).astype(int), 0, n - 1)
    for k in range(n):
        u, t = np.unique(T[sector == k], return_inverse=True)
        io.write_tri(str(d / f"s{k}.tri"), .6 * V[u], t.reshape(-1, 3))
    for name, r in (("skull", .8), ("scalp", 1.0)):
        io.write_tri(str(d / f"{name}.tri"), r * V, T)
    (d / "h.geom").write_text(
        f"# Domain Description 1.1\n\nMeshes {n + 2}\n" + "".join(f'Mesh s{k}: "s{k}.tri"\n' for k in range(n)) +
        'Mesh skull: "skull.tri"\nMesh scalp: "scalp.tri"\n\nInterfaces 3\n\nInterface In: ' + " ".join(f"s{k}" for k in range(n)) +
        "\nInterface Skull: skull\nInterface Scalp: scalp\n\nDomains 4\n\nDomain BRAIN: -In\nDomain SKULL: +In -Skull\n"
        "Domain SCALP: +Skull -Scalp\nDomain AIR: +Scalp\n")
    (d / "h.cond").write_text("# Properties Description 1.0 (Conductivities)\n\nAIR 0.0\nBRAIN 1\nSKULL 0.1\nSCALP 1\n")
    return api.Geometry(str(d / "h.geom"), str(d / "h.cond"))


def test_mixed_gain_is_the_fp64_gain(geo):
    from openmeeg_gb300 import api, synthetic as syn
    dip = syn.random_dipoles(20, 5, .5)
    dip[10:, :3] *= (.7 / np.linalg.norm(dip[10:, :3], axis=1))[:, None]   # half of them in the next shell
    el = syn.fibonacci_points(12, 1.0)
    a = api.forward_gain(geo, dip, el, None, precision="fp64")[0].cpu().numpy()
    b = api.forward_gain(geo, dip, el, None, precision="mixed")[0].cpu().numpy()
    assert np.max(np.linalg.norm(a - b, axis=0) / np.linalg.norm(a, axis=0)) < 1e-5


def test_points_inside(geo):
    from openmeeg_gb300 import api, synthetic as syn
    p = syn.random_dipoles(60, 6, .55)[:, :3]
    S = api.Surf2VolMat(geo, p)
    assert S.shape[0] == 60
    q = syn.random_dipoles(1, 7, .3)
    P = api.DipSource2InternalPotMat(geo, q, p).cpu().numpy()[:, 0]
    x = p - q[0, :3]
    want = x @ q[0, 3:] / (4 * np.pi * np.linalg.norm(x, axis=1)**3)   # the source's own domain, sigma 1
    assert rel(P, want) < 1e-12
