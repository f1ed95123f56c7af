"""The S / D tables' block fixed point and batches against the oracle.

Lengths of 1e-3 and 1e3 and a head far from the origin (every exponent of the
fixed-point vectors moves), and a surface whose tables take two batches, the
second of which starts its triangles in another order.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _head(scale, shift, fine):
    from openmeeg_gb300 import synthetic as syn
    meshes = [syn.icosphere(fine), syn.icosphere(1), syn.icosphere(0)]
    domains = [("in", [-1], 1.0), ("mid", [1, -2], 0.0125), ("out", [2, -3], 0.7), ("Air", [3], 0.0)]
    V = [scale * (r * v + np.asarray(shift)) for (v, t), r in zip(meshes, (0.3, 0.6, 1.0))]
    return syn.NestedHead(V, [t for v, t in meshes], ["a", "b", "c"], domains)


@pytest.mark.parametrize("scale,shift,fine", [(1e-3, (0, 0, 0), 1), (1e3, (0, 0, 0), 1), (1.0, (50.0, -20.0, 7.0), 1),
                                              (1.0, (0, 0, 0), 3)])
def test_head_matrix_matches_oracle(cuda, scale, shift, fine):
    from openmeeg_gb300 import api
    from oracle import oracle
    head = _head(scale, shift, fine)
    ref = oracle.headmat(oracle.digest(head))
    hm = api.HeadMat(api.Geometry.from_head(head)).cpu().numpy()
    # the parity bound of the FP64 head matrix
    assert np.linalg.norm(hm - ref) <= 1e-12 * np.linalg.norm(ref)
