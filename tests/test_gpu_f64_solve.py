"""FP64 solver (digit factorization and sweeps) against LAPACK on small quasi-definite systems."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(sub, layers):
    from openmeeg_gb300 import api, workloads
    w = workloads.small(sub, layers=layers, perturb=True)
    geo = api.Geometry.from_head(w.head)
    return geo, api.HeadMat(geo).cpu().numpy()


# sizes around the 64 / 128 / 256 blocks: 166, 292 and 1126 (3 layers), 1608 (4 layers) unknowns
@pytest.mark.parametrize("sub,layers", [(0, 3), (1, 3), (1, 4), (2, 3), (2, 4)])
@pytest.mark.parametrize("nrhs", [1, 2, 63, 131])
def test_solve_matches_lapack(cuda, sub, layers, nrhs):
    from openmeeg_gb300 import api
    geo, hm = _system(sub, layers)
    n = hm.shape[0]
    rng = np.random.default_rng(nrhs)
    x = rng.standard_normal((n, nrhs)) * np.exp(4 * rng.standard_normal((1, nrhs)))
    b = hm @ x
    got = api.Solver(geo, hm=hm).solve(b).cpu().numpy()
    ref = np.linalg.solve(hm, b)
    # forward error bound of a backward stable solve: n eps cond, per column
    bound = n * 2.0**-52 * np.linalg.cond(hm)
    assert np.all(np.linalg.norm(got - x, axis=0) <= bound * np.linalg.norm(x, axis=0))
    # and no further off than LAPACK's own by more than a small factor
    assert np.linalg.norm((got - x) / np.linalg.norm(x, axis=0)) <= 10 * np.linalg.norm(
        (ref - x) / np.linalg.norm(x, axis=0)) + 1e-13


def test_solve_many_right_hand_sides_in_parts(cuda):
    """Columns are independent of the others solved with them."""
    import torch
    from openmeeg_gb300 import api
    geo, hm = _system(1, 3)
    sv = api.Solver(geo, hm=hm)
    b = np.random.default_rng(1).standard_normal((hm.shape[0], 300))
    whole = sv.solve(b)
    parts = torch.cat([sv.solve(b[:, :7]), sv.solve(b[:, 7:150]), sv.solve(b[:, 150:])], 1)
    assert torch.equal(whole, parts)
