"""Gains whose sources touch more runs of rows than one launch lists.

A brain with four two-shell inclusions, numbered outer, inner, outer, inner ...:
dipoles in the brain have rows on the four outer shells and the brain's surface,
five runs of meshes that are not adjacent, ten ranges of rows.  FP64 against the
oracle at 1e-10 as the other gains, mixed precision at the 1e-6 of its refinement.
"""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


def _head():
    from openmeeg_gb300 import synthetic as syn
    V0, T0 = syn.icosphere(1)
    V, T, dom = [], [], []
    for k, c in enumerate([(.45, 0, 0), (-.45, 0, 0), (0, .45, 0), (0, -.45, 0)]):
        V += [np.array(c) + .2 * V0, np.array(c) + .1 * V0]
        T += [T0, T0]
        dom += [(f"shell{k}", [-(2 * k + 1), 2 * k + 2], .3), (f"core{k}", [-(2 * k + 2)], 1.5)]
    V += [.87 * V0, .92 * V0, V0]
    T += [T0, T0, T0]
    dom += [("brain", [-9, 1, 3, 5, 7], 1.0), ("skull", [9, -10], .0125), ("scalp", [10, -11], 1.0), ("air", [11], 0.0)]
    return syn.NestedHead(V, T, [f"m{k}" for k in range(11)], dom)


@pytest.fixture(scope="module")
def case(cuda):
    from openmeeg_gb300 import synthetic as syn
    from oracle import oracle
    head = _head()
    dip = syn.random_dipoles(40, 3, 0.7)
    r = np.min([np.linalg.norm(dip[:, :3] - c, axis=1) for c in
                [(.45, 0, 0), (-.45, 0, 0), (0, .45, 0), (0, -.45, 0)]], axis=0)
    dip = dip[r > .25]
    ele, sq = syn.fibonacci_points(16, 1.0), syn.radial_magnetometers(9, 1.2)
    g = oracle.digest(head)
    HM, D = oracle.headmat(g), oracle.dsm(g, dip)
    return (head, dip, ele, sq, oracle.gain_eeg(HM, D, oracle.h2em(g, ele)),
            oracle.gain_meg(HM, D, oracle.h2mm(g, sq), oracle.ds2mm(dip, sq)))


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-6)])
@pytest.mark.parametrize("which", ["both", "eeg", "meg"])
def test_gain(case, precision, tol, which):
    from openmeeg_gb300 import api
    head, dip, ele, sq, e, m = case
    geo = api.Geometry.from_head(head)
    ge, gm, _ = api.forward_gain(geo, dip, None if which == "meg" else ele, None if which == "eeg" else sq,
                                 precision=precision)
    if which != "meg":
        assert rel(ge.cpu().numpy(), e) < tol
    if which != "eeg":
        assert rel(gm.cpu().numpy(), m) < tol


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-6)])
def test_batch(case, precision, tol):
    from openmeeg_gb300 import api
    head, dip, ele, sq, e, m = case
    b = api.BatchForward([(api.Geometry.from_head(head), dip, ele, sq)] * 2, precision=precision)
    b.run()
    for i in range(2):
        ge, gm = b.gains(i)
        assert rel(ge.cpu().numpy(), e) < tol and rel(gm.cpu().numpy(), m) < tol
