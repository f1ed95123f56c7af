"""The integer-pipe square root, edge logarithm and half solid angle against 60 digits.

Arguments on both sides of every polynomial's limit, powers of two and their
neighbours (where the residual of the approximate reciprocal changes scale),
mantissas of all ones, and what no polynomial takes.  Error bound: the rounding,
2^-53, and at most four products of 60 bits, 2 units each, and the residual's
third order, 2^-58.8: under 2^-56 together.  Beyond 1/2 a few roundings of the
sums that the argument is reduced by: 2^-50.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TIGHT, REDUCED = 2.0 ** -53 * 1.125, 2.0 ** -50


def _eval(which, a, b, wr=0.0):
    import torch
    from openmeeg_gb300 import _lib
    f = _lib.load().omg_internal_fixed64
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int, ctypes.c_int64, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_double, ctypes.c_void_p]
    a, b = (torch.as_tensor(np.asarray(v, np.float64), device="cuda") for v in (a, b))
    out = torch.empty_like(a)
    assert f(which, a.numel(), a.data_ptr(), b.data_ptr(), wr, out.data_ptr()) == 0
    return out.cpu().numpy()


def _values(n, rng):
    one = [1.0, np.nextafter(1, 2), np.nextafter(2, 1), 1.5, 1 + 2.0 ** -21, 2 - 2.0 ** -21, 2.0 ** 0.5]
    v = np.concatenate([one, 1 + rng.random(n - len(one))])
    return np.ldexp(v, rng.integers(-60, 60, n))


@pytest.mark.parametrize("n", [1, 31, 400])
def test_square_root(cuda, n):
    mp = pytest.importorskip("mpmath").mp
    mp.dps = 60
    a = _values(max(n, 8), np.random.default_rng(n))[:n]
    for x, y in zip(a, _eval(0, a, a)):
        r = mp.sqrt(mp.mpf(float(x)))
        assert abs(mp.mpf(float(y)) / r - 1) <= TIGHT, float(x)


@pytest.mark.parametrize("n", [1, 31, 400])
@pytest.mark.parametrize("which", [3, 4])
def test_reciprocal_square_root(cuda, n, which):
    mp = pytest.importorskip("mpmath").mp
    mp.dps = 60
    wr = 0.027230314174434
    a = _values(max(n, 8), np.random.default_rng(n))[:n]
    for x, y in zip(a, _eval(which, a, a, wr)):
        r = (mp.mpf(wr) if which == 4 else 1) / mp.sqrt(mp.mpf(float(x)))
        assert abs(mp.mpf(float(y)) / r - 1) <= TIGHT, float(x)
    with np.errstate(all="ignore"):
        end = _eval(which, [0.0, np.inf, np.nan, -1.0], [0.0] * 4, wr)
    assert np.isinf(end[0]) and end[1] == 0.0 and np.isnan(end[2:]).all()


@pytest.mark.parametrize("which", [1, 2])
@pytest.mark.parametrize("wr", [0.0, 0.027230314174434, 0.333333333333334])
@pytest.mark.parametrize("lo,hi", [(1e-9, 2.0 ** -7), (0.99 / 16, 1.01 / 16), (0.99 / 8, 1.01 / 8), (0.2, 0.3),
                                   (0.4999, 0.5001), (0.5, 0.999)])
def test_edge_and_angle(cuda, which, wr, lo, hi):
    mp = pytest.importorskip("mpmath").mp
    mp.dps = 60
    rng = np.random.default_rng(3)
    a = _values(150, rng)
    b = a * rng.uniform(lo, hi, 150)
    if which == 2:
        b *= rng.choice([-1.0, 1.0], 150)
    for x, z, y in zip(a, b, _eval(which, a, b, wr)):
        X, Z = mp.mpf(float(x)), mp.mpf(float(z))
        r = (2 * mp.atanh(Z / X) / Z if which == 1 else mp.atan2(Z, X)) * mp.mpf(wr if wr else 1.0)
        tol = TIGHT if abs(z) < 0.4999999 * x else REDUCED
        assert abs(mp.mpf(float(y)) / r - 1) <= tol, (float(x), float(z))


@pytest.mark.parametrize("wr", [0.0, 0.027230314174434])
def test_every_quadrant(cuda, wr):
    mp = pytest.importorskip("mpmath").mp
    mp.dps = 60
    rng = np.random.default_rng(4)
    t = np.concatenate([np.tan(np.arange(-16, 17) * np.pi / 16 + 1e-9), [2.0, 0.5, 1.0, -1.0, -2.0, -0.5],
                        np.ldexp(rng.uniform(-1, 1, 300), rng.integers(-8, 9, 300))])
    a = _values(len(t), rng) * rng.choice([-1.0, 1.0], len(t))
    b = a * t
    for x, z, y in zip(a, b, _eval(2, a, b, wr)):
        r = mp.atan2(mp.mpf(float(z)), mp.mpf(float(x))) * mp.mpf(wr if wr else 1.0)
        assert abs(mp.mpf(float(y)) / r - 1) <= REDUCED, (float(x), float(z))


@pytest.mark.parametrize("wr", [0.0, 0.027230314174434])
def test_points_close_to_an_edge(cuda, wr):
    mp = pytest.importorskip("mpmath").mp
    mp.dps = 60
    rng = np.random.default_rng(5)
    b = _values(300, rng)
    a = b * (1 + np.ldexp(rng.uniform(0.5, 1, 300), rng.integers(-50, 1, 300)))
    for x, z, y in zip(a, b, _eval(1, a, b, wr)):
        X, Z = mp.mpf(float(x)), mp.mpf(float(z))
        r = mp.log((X + Z) / (X - Z)) / Z * mp.mpf(wr if wr else 1.0)
        assert abs(mp.mpf(float(y)) / r - 1) <= REDUCED, (float(x), float(z))


def test_values_no_polynomial_takes(cuda):
    inf, nan = np.inf, np.nan
    with np.errstate(all="ignore"):
        assert np.array_equal(_eval(0, [0.0, inf, 1e-310], [0.0] * 3), np.sqrt([0.0, inf, 1e-310]))
        assert np.isnan(_eval(0, [nan, -1.0], [0.0] * 2)).all()
        a = [0.0, -1.0, -1.0, 0.0, inf, 3.0, 3.0, -2.0, 1.0]
        b = [1.0, 0.0, -1.0, -2.0, 1.0, 0.0, inf, 5.0, 7.0]
        assert np.allclose(_eval(2, a, b), np.arctan2(b, a), rtol=1e-15, atol=0)
    assert np.isnan(_eval(2, [nan, 1.0, nan], [1.0, nan, 0.0])).all()
    assert np.isnan(_eval(1, [nan, 1.0, nan], [1.0, nan, 0.5])).all()
    assert np.isinf(_eval(1, [3.0], [3.0])).all()
