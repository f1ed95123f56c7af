"""The digit products hold FP64's own error bounds.

General products (omg_gemm_f64_dev): K 2^-53 sum |a||b| for every entry, as FP64
multiply-adds, also where a row's entries span many powers of two (few such entries:
a CTA each; many: FP64 tiles), and in norm no larger an error than FP64
multiply-adds make on rows with peaks, which is what potentials and sources are.
Updates: digits of the largest magnitude, against Python's integers.  Other truths in
np.longdouble (64 bits and more).
"""
import ctypes

import numpy as np
import pytest

from test_gpu_f64_gemm import _gemm

pytestmark = pytest.mark.gpu
L = np.longdouble


def _check(A, B, C, out, alpha, beta, rows=None):
    """K 2^-53 sum |a||b| for the product, its sum over segments and with beta C."""
    K = A.shape[1]
    want = alpha * (A.astype(L) @ B.astype(L)) + beta * C.astype(L)
    mag = np.abs(A) @ np.abs(B)
    bound = 2.0**-53 * ((K + 4) * abs(alpha) * mag + 2 * np.abs(beta * C) + 2 * np.abs(want).astype(float))
    assert np.all(np.abs(out - want).astype(float) <= bound)


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("spread,M,N,K", [(1.0, 70, 90, 700), (4.0, 129, 33, 513), (8.0, 33, 65, 1000), (16.0, 65, 31, 257),
                                          (8.0, 1, 1, 3000), (3.0, 300, 257, 600)])
def test_graded_operands(cuda, ta, tb, spread, M, N, K):
    rng = np.random.default_rng(M + N + K)
    A = rng.standard_normal((M, K)) * np.exp(spread * rng.standard_normal((M, K)))
    B = rng.standard_normal((K, N)) * np.exp(spread * rng.standard_normal((K, N)))
    C = rng.standard_normal((M, N))
    for alpha, beta in ((1.0, 0.0), (-0.5, 3.0)):
        _check(A, B, C, _gemm(cuda, A, B, C, ta, tb, alpha, beta, 1), alpha, beta)


@pytest.mark.parametrize("ta", [0, 1])
def test_few_graded_entries_and_zero_rows(cuda, ta):
    """One row against one column far from its peak, rows and segments of zeros, values next to the subnormals."""
    rng = np.random.default_rng(8)
    A, B = rng.standard_normal((200, 800)), rng.standard_normal((800, 150))
    A[7, :600], A[9], B[:600, 11], B[300:, 20] = 1e-30 * A[7, :600], 0.0, 0.0, 0.0
    A[7, 700], B[700, 13] = 1e12, 0.0
    A[50] *= 2.0**-700
    B[:, 60] *= 2.0**-340   # (their product's terms are about 2^-1040)
    C = np.zeros((200, 150))
    out = _gemm(cuda, A, B, C, ta, 0, 1.0, 0.0, 0)
    tiny = out[50, 60]
    out[50, 60] = float(A[50].astype(L) @ B[:, 60].astype(L))
    _check(A, B, C, out, 1.0, 0.0)
    assert abs(tiny - out[50, 60]) <= 800 * 2.0**-1074   # FP64 underflows term by term
    assert np.all(out[9] == 0.0)


def test_rows_with_peaks(cuda):
    """Kernels like 1/r against dipole-like columns: the error is below that of multiply-adds in K order."""
    rng = np.random.default_rng(3)
    K, M, N = 3000, 40, 60
    z = rng.random(K)
    r = np.abs(z[None] - rng.random((M, 1)))
    A = 1.0 / (r + 1e-3)
    d = z[:, None] - rng.random((1, N))
    B = d / (d**2 + 1e-4)**1.5
    want = A.astype(L) @ B.astype(L)
    fma = np.zeros((M, N))
    for k in range(K):
        fma = (fma.astype(L) + A[:, k:k + 1].astype(L) * B[k].astype(L)).astype(float)
    out = _gemm(cuda, A, B, np.zeros((M, N)), 1, 0, 1.0, 0.0, 0)
    err = lambda x, axis: np.linalg.norm(np.abs(x - want).astype(float), axis=axis)
    for axis in (None, 0, 1):
        assert np.all(err(out, axis) <= err(fma, axis))


@pytest.mark.parametrize("M,N,K", [(116500, 3, 300), (2, 116600, 400), (7700, 7700, 130), (1, 1, 17_000_000)])
def test_sizes_past_one_block(cuda, M, N, K):
    """Rows, columns and output past one block of the scratch, and more segments than a grid's second dimension holds."""
    import torch
    from openmeeg_gb300 import _lib, api
    g = torch.Generator(device=cuda).manual_seed(1)
    A = torch.randn(M, K, dtype=torch.float64, device=cuda, generator=g)   # op(A) = A by its transpose
    B = torch.randn(N, K, dtype=torch.float64, device=cuda, generator=g)
    C = torch.empty(N, M, dtype=torch.float64, device=cuda)
    ctx, p = api.Context.default(), lambda t: ctypes.c_void_p(t.data_ptr())
    _lib.check(ctx.lib.omg_gemm_f64_dev(ctx.handle, 1, 0, M, N, K, 1.0, p(A), K, p(B), K, 0.0, p(C), M))
    i = np.unique(np.r_[np.arange(min(M, 3)), M // 2, np.arange(max(M - 3, 0), M)])
    j = np.unique(np.r_[np.arange(min(N, 3)), N // 2, np.arange(max(N - 3, 0), N)])
    a, b = A.cpu().numpy()[i], B.cpu().numpy()[j].T
    out = C.cpu().numpy().T[np.ix_(i, j)]
    want = a.astype(L) @ b.astype(L)
    mag = np.abs(a) @ np.abs(b)
    assert np.all(np.abs(out - want).astype(float) <= 2.0**-53 * (min(K, 512) * mag + 2 * np.abs(want).astype(float)))
    full = A @ B.T if M * N < 10**8 else None
    if full is not None:   # every block was written
        assert float((C.T - full).abs().max()) < 1e-9 * K**0.5


def _update(cuda, A, B):
    import torch
    from openmeeg_gb300 import _lib
    M, k = A.shape
    N = B.shape[0]
    f = _lib.load().omg_internal_digit_update
    f.restype, f.argtypes = ctypes.c_int, [ctypes.c_int64, ctypes.c_int64, ctypes.c_int] + [ctypes.c_void_p] * 3 + [
        ctypes.c_int, ctypes.c_void_p]
    da, db = (torch.as_tensor(np.ascontiguousarray(x.T), device=cuda) for x in (A, B))
    C, err = torch.zeros(N, M, dtype=torch.float64, device=cuda), torch.zeros(4, dtype=torch.int32, device=cuda)
    torch.cuda.synchronize()
    assert f(M, N, k, da.data_ptr(), db.data_ptr(), C.data_ptr(), 0, err.data_ptr()) == 0 and not err.any()
    return -C.T.cpu().numpy()


@pytest.mark.parametrize("first", [100, -100])
@pytest.mark.parametrize("rest", [-128, -127, 127])
def test_update_with_all_digits_large(cuda, first, rest):
    """Digits of the largest magnitude in every place: the levels' sums reach their 2^24."""
    Z = first * 2**48 + rest * sum(2**(8 * j) for j in range(6))
    if rest == 127 and first < 0:   # (magnitudes next to each other, of both signs)
        Z = first * 2**48 - 127 * sum((-1)**j * 2**(8 * j) for j in range(6))
    x = float(Z >> 3) * 2.0**-53 if Z % 8 == 0 else float(Z) * 2.0**-56
    digits = int(x * 2.0**56)   # what FP64 holds of it
    A, B = np.full((140, 256), x), np.full((70, 256), x)
    B[::2] = -B[::2]
    got = _update(cuda, A, B)
    want = float(256 * digits * digits / 2**112)
    # sums past 2^24 round in the accumulators, to 16 units of level 6 at most
    assert np.all(np.abs(got[:, 1::2] - want) <= 16 * 2.0**-48 + 2.0**-53 * abs(want))
    assert np.all(np.abs(got[:, ::2] + want) <= 16 * 2.0**-48 + 2.0**-53 * abs(want))
