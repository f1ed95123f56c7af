"""FP64-accurate digit products and the 32-column panel kernel of the FP64 factorization.

The digits keep 56 bits below each row's maximum and all digit pairs down to 2^-58 of
the product of the row maxima, so an entry of C - A B^T is off by at most
2^-54 K max|A_i.| max|B_j.| from them and by one rounding of the result; the tests
allow 2^-52 of both (the bound of an FP64 product over K terms is 2^-53 K).
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lib():
    from openmeeg_gb300 import _lib
    lib = _lib.load()
    lib.omg_internal_digit_update.argtypes = [ctypes.c_int64, ctypes.c_int64, ctypes.c_int] + [ctypes.c_void_p] * 3 + [
        ctypes.c_int, ctypes.c_void_p]
    lib.omg_internal_panel32.argtypes = [ctypes.c_int, ctypes.c_int64] + [ctypes.c_void_p] * 3
    return lib


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _update(cuda, A, B, C, lower):
    """C - A B^T by the kernel (A: M x k, B: Nc x k, C: M x Nc numpy)."""
    import torch
    a, b, c = (torch.as_tensor(np.ascontiguousarray(x.T)).to(cuda) for x in (A, B, C))
    err = torch.zeros(4, dtype=torch.int32, device=cuda)
    torch.cuda.synchronize()
    assert _lib().omg_internal_digit_update(A.shape[0], B.shape[0], A.shape[1], _p(a), _p(b), _p(c), lower, _p(err)) == 0
    assert int(err[0]) == 0
    return c.cpu().numpy().T


def _check(out, A, B, C, lower):
    ref = C.astype(np.longdouble) - A.astype(np.longdouble) @ B.astype(np.longdouble).T
    bound = 2.0**-52 * (A.shape[1] * np.abs(A).max(1)[:, None] * np.abs(B).max(1)[None] + np.abs(C))
    live = np.tril(np.ones(C.shape, bool)) if lower else np.ones(C.shape, bool)
    assert np.all(np.abs(out - ref).astype(float)[live] <= bound[live])
    assert np.array_equal(out[~live], C[~live])


@pytest.mark.parametrize("M,Nc,k,lower", [(1, 1, 1, 0), (128, 128, 128, 0), (130, 77, 100, 0), (127, 257, 256, 0),
                                          (300, 300, 256, 1), (129, 129, 129, 1), (1700, 1700, 128, 1)])
def test_digit_update(cuda, M, Nc, k, lower):
    rng = np.random.default_rng(M + Nc + k)
    A = rng.standard_normal((M, k)) * np.exp(3 * rng.standard_normal((M, 1))) * np.exp(rng.standard_normal((1, k)))
    B = A if lower else rng.standard_normal((Nc, k)) * np.exp(3 * rng.standard_normal((Nc, 1)))
    C = rng.standard_normal((M, Nc))
    _check(_update(cuda, A, B, C, lower), A, B, C, lower)


def test_digit_update_extreme_digits(cuda):
    """Entries whose digits all have the largest magnitude, zero rows, and entries far below their row's maximum."""
    x = -128.0 * sum(2.0 ** (8 * j) for j in range(7)) * 2.0**-56
    A = np.full((140, 256), x)
    A[3] = 0.0
    A[5, 1:] *= 2.0**-40
    A[7] *= 2.0**300
    A[8] *= 2.0**-300
    B = A[:70] * np.where(np.arange(256) % 3 == 0, 1.0, -1.0)
    C = np.zeros((140, 70))
    out = _update(cuda, A, B, C, 0)
    _check(out, A, B, C, 0)
    assert np.all(out[3] == 0.0) and np.all(out[:, 3] == 0.0)


def test_digit_update_not_finite_rows(cuda):
    rng = np.random.default_rng(0)
    A, B, C = rng.standard_normal((40, 64)), rng.standard_normal((30, 64)), rng.standard_normal((40, 30))
    A[4, 10], B[7, 3] = np.nan, np.inf
    out = _update(cuda, A, B, C, 0)
    bad = np.zeros(C.shape, bool)
    bad[4], bad[:, 7] = True, True
    assert np.all(np.isnan(out[bad]))
    ok = [i for i in range(40) if i != 4], [j for j in range(30) if j != 7]
    _check(out[np.ix_(*ok)], A[ok[0]], B[ok[1]], C[np.ix_(*ok)], 0)


def _panel(cuda, A, P):
    """The factor of A and the rows P L^-T by the kernel (w x w, m x w numpy), its status and column."""
    import torch
    w, m = A.shape[0], P.shape[0]
    a = torch.as_tensor(np.ascontiguousarray(np.vstack([A, P]).T)).to(cuda)
    err, col = torch.zeros(4, dtype=torch.int32, device=cuda), torch.zeros(1, dtype=torch.int64, device=cuda)
    torch.cuda.synchronize()
    assert _lib().omg_internal_panel32(w, m, _p(a), _p(err), _p(col)) == 0
    out = a.cpu().numpy().T
    return np.tril(out[:w]), out[w:], int(err[0]), int(col[0])


@pytest.mark.parametrize("w,m", [(1, 0), (2, 0), (31, 0), (32, 0), (32, 1), (32, 33), (32, 300)])
def test_panel(cuda, w, m):
    rng = np.random.default_rng(w + m)
    X = rng.standard_normal((w, w))
    A, P = X @ X.T + w * np.eye(w), rng.standard_normal((m, w))
    L, W, status, _ = _panel(cuda, A, P)
    assert status == 0
    # Cholesky's and the substitution's backward error, w eps
    assert np.linalg.norm(L @ L.T - A) <= 2.0**-52 * w * np.linalg.norm(A)
    assert np.linalg.norm(W @ L.T - P) <= 2.0**-52 * w * np.linalg.norm(W) * np.linalg.norm(L)


@pytest.mark.parametrize("per_sm,more", [(8, 0), (8, 1), (16, 0), (16, 3), (32, 5)])
def test_panel_rows_per_cta(cuda, per_sm, more):
    """Both sides of the numbers of rows at which a row takes 16, 8 and 4 lanes."""
    import torch
    m = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    rng = np.random.default_rng(m)
    X = rng.standard_normal((32, 32))
    A, P = X @ X.T + 32 * np.eye(32), rng.standard_normal((m, 32))
    L, W, status, _ = _panel(cuda, A, P)
    assert status == 0
    # the substitution's backward error, w eps
    assert np.linalg.norm(W @ L.T - P) <= 2.0**-52 * 32 * np.linalg.norm(W) * np.linalg.norm(L)


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_panel_reports_entries_that_are_not_finite(cuda, value):
    A = 4.0 * np.eye(32)
    A[12, 5] = A[5, 12] = value
    assert _panel(cuda, A, np.ones((3, 32)))[2] == -3


def test_panel_reports_the_wrong_sign(cuda):
    A = np.eye(32)
    A[9, 9] = -1.0
    A[20, 20] = np.nan
    assert _panel(cuda, A, np.zeros((1, 32)))[2:] == (-3, 9)
