"""omg_gemm_f64_dev over its forms: transposes, sizes on both sides of the digit products' rule, beta, not finite entries."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gemm(cuda, A, B, C, ta, tb, alpha, beta, pad):
    """alpha op(A) op(B) + beta C by the library; op(A): M x K, op(B): K x N given as numpy, stored column-major with
    leading dimensions `pad` beyond the rows."""
    import torch
    from openmeeg_gb300 import api
    ctx = api.Context.default()

    def store(X):   # column-major buffer with a longer leading dimension
        t = torch.full((X.shape[1], X.shape[0] + pad), np.nan, dtype=torch.float64)
        t[:, :X.shape[0]] = torch.as_tensor(np.ascontiguousarray(X.T))
        return t.to(cuda)

    a, b, c = store(A.T if ta else A), store(B.T if tb else B), store(C)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    torch.cuda.synchronize()
    api.check(ctx.lib.omg_gemm_f64_dev(ctx.handle, int(ta), int(tb), C.shape[0], C.shape[1], A.shape[1], alpha, p(a),
                                       a.shape[1], p(b), b.shape[1], beta, p(c), c.shape[1]))
    out = c.cpu().numpy().T
    assert np.all(np.isnan(out[C.shape[0]:]))
    return out[:C.shape[0]]


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (40, 30, 100), (33, 7, 255), (215, 8, 257), (130, 129, 1000), (5, 3000, 300),
                                   (1, 1, 5000)])
def test_gemm(cuda, ta, tb, M, N, K):
    rng = np.random.default_rng(M + N + K)
    A = rng.standard_normal((M, K)) * np.exp(2 * rng.standard_normal((M, 1)))
    B = rng.standard_normal((K, N)) * np.exp(2 * rng.standard_normal((1, N)))
    C = rng.standard_normal((M, N))
    ref = A.astype(np.longdouble) @ B.astype(np.longdouble)
    rows = np.abs(A).max(1)[:, None] * np.abs(B).max(0)[None]
    for alpha, beta in ((1.0, 0.0), (-0.5, 1.0), (2.0, -3.0)):
        out = _gemm(cuda, A, B, C, ta, tb, alpha, beta, 3)
        want = alpha * ref + beta * C
        # the digits' 2^-54 K max max, the FP64 kernel's 2^-53 K |A||B|, the sum over the K / 256 segments, the result
        bound = 2.0**-52 * (abs(alpha) * rows * K * (1 + K / 512) + np.abs(beta * C) + np.abs(want).astype(float))
        assert np.all(np.abs(out - want).astype(float) <= bound)


def test_gemm_not_finite(cuda):
    """Infinities and NaN come out where IEEE arithmetic puts them, on the digit path too."""
    rng = np.random.default_rng(5)
    A, B = rng.standard_normal((60, 700)), rng.standard_normal((700, 50))
    A[3, 10], A[9, 600], B[300, 7], B[20, 8] = np.inf, np.nan, -np.inf, np.inf
    B[10, 5] = 0.0
    with np.errstate(invalid="ignore"):
        want = A @ B
    out = _gemm(cuda, A, B, np.zeros((60, 50)), 0, 0, 1.0, 0.0, 0)
    assert np.array_equal(np.isnan(out), np.isnan(want))
    assert np.array_equal(out[np.isinf(want)], want[np.isinf(want)])
    ok = np.isfinite(want)
    assert np.all(np.isfinite(out[ok])) and np.allclose(out[ok], want[ok], rtol=0, atol=1e-11)
