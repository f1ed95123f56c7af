"""SurfSourceMat of a source surface past the 65535 CTAs of a grid's second dimension.

A sheet of triangles inside the innermost sphere; a vertex's column depends on its
own triangles alone, so the columns of small pieces cut from the sheet's ends and
middle are the sheet's: to the 1e-13 by which the order of a vertex's triangles and
the polynomial that a warp's 32 triangles share may differ.  Two sheets: past
131070 triangles (two per CTA of the pairs), and past 262140 and 524280 vertices.
"""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


def _sheet(n, m):
    x, y = np.meshgrid(np.linspace(-.3, .3, n), np.linspace(-.3, .3, m), indexing="ij")
    V = np.stack([x, y, .1 + .1 * np.sin(4 * x) * np.cos(3 * y)], -1).reshape(-1, 3)
    i = (np.arange(n - 1)[:, None] * m + np.arange(m - 1)).ravel()
    T = np.concatenate([np.stack([i, i + m, i + 1], 1), np.stack([i + 1, i + m, i + m + 1], 1)])
    return V, T[np.argsort(T.min(1), kind="stable")]


@pytest.mark.parametrize("n,m", [(260, 256), (740, 712)])
def test_columns_of_a_large_sheet(cuda, n, m):
    import torch
    from openmeeg_gb300 import api, synthetic as syn
    head = syn.nested_head(0, [.8, .9, 1.0], [1.0, .0125, 1.0])
    geo = api.Geometry.from_head(head)
    V, T = _sheet(n, m)
    assert len(T) > (131070 if n < 300 else 1048560)
    S = api.SurfSourceMat(geo, V, T)
    for r in (0, n // 2, n - 5):   # five rows of the sheet
        lo, hi = r * m, (r + 5) * m
        t = T[((T >= lo) & (T < hi)).all(1)] - lo
        part = api.SurfSourceMat(geo, V[lo:hi], t)
        inner = slice(m, 4 * m)   # vertices with all their triangles
        a, b = S[:, lo:hi][:, inner], part[:, inner]
        assert float(b.abs().max()) > 0
        assert rel(a.cpu().numpy(), b.cpu().numpy()) < 1e-13
    torch.cuda.empty_cache()
