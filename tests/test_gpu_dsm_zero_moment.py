"""Dipoles of no moment have columns of zeros (their moment has no exponent to cut digits by)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,levels,tol", [(3, 10, 1e-3), (3, 0, 1e-3), (0, 3, 0.0)])
def test_columns_of_zeros(cuda, order, levels, tol):
    from openmeeg_gb300 import _lib, api, workloads
    w = workloads.small(1, layers=3)
    d = np.array(w.dipoles[:5])
    d[1, 3:] = 0.0
    d[3, 3:] = -0.0
    D = api.DipSourceMat(api.Geometry.from_head(w.head), d, _lib.Integrator(order, levels, tol)).cpu().numpy()
    assert np.all(D[:, [1, 3]] == 0.0) and np.all(np.any(D[:, [0, 2, 4]] != 0.0, axis=0))
