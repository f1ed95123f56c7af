"""The shared-table S / D kernels of the FP64 head matrix against the oracle.

Nested boxes (coplanar triangles: heights and solid angles that vanish; right
angles; points close to neighbours' edges) and a sphere inside a box, at triangle
counts off the warp and batch sizes, with every rule of the integrator.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _box(n, half):
    """Surface of a cube: 6 n^2 squares of two triangles, shared vertices, inward normals."""
    V, T, at = [], [], {}

    def vert(p):
        if p not in at:
            at[p] = len(V)
            V.append([half * (2.0 * c / n - 1.0) for c in p])
        return at[p]

    for axis in range(3):
        for side in (0, n):
            for i in range(n):
                for j in range(n):
                    def corner(a, b):
                        p = [0, 0, 0]
                        p[axis], p[(axis + 1) % 3], p[(axis + 2) % 3] = side, a, b
                        return vert(tuple(p))
                    q = [corner(i, j), corner(i + 1, j), corner(i + 1, j + 1), corner(i, j + 1)]
                    if side == n:   # outward is counter-clockwise here: turn it
                        q = q[::-1]
                    T += [[q[0], q[1], q[2]], [q[0], q[2], q[3]]]
    return np.array(V), np.array(T, np.int64)


def _head(kind):
    from openmeeg_gb300 import synthetic as syn
    if kind == "boxes":
        meshes = [_box(2, 0.6), _box(3, 0.8), _box(3, 1.0)]
    else:
        v, t = syn.icosphere(1)
        meshes = [(0.5 * v, t), _box(4, 0.7), _box(2, 1.0)]
    domains = [("in", [-1], 1.0), ("mid", [1, -2], 0.0125), ("out", [2, -3], 0.7), ("Air", [3], 0.0)]
    return syn.NestedHead([m[0] for m in meshes], [m[1] for m in meshes], ["a", "b", "c"], domains)


@pytest.mark.parametrize("kind", ["boxes", "sphere_in_box"])
@pytest.mark.parametrize("order", [0, 1, 2, 3])
def test_head_matrix_of_boxes_matches_oracle(cuda, kind, order):
    from openmeeg_gb300 import api
    from oracle import oracle
    head = _head(kind)
    ref = oracle.headmat(oracle.digest(head), order=order)
    hm = api.HeadMat(api.Geometry.from_head(head), integrator=api.Integrator(order, 0, 0.005)).cpu().numpy()
    # the parity bound of the FP64 head matrix
    assert np.linalg.norm(hm - ref) <= 1e-12 * np.linalg.norm(ref)
