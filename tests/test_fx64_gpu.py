"""The digit products and factorizations of fx64.cu at the edges of their tiles (32-wide
steps, 64 x 128 output tiles, 128-row blocks, 128- to 512-wide panels) against extended
precision.

Product: each entry is rounded within 2^-61 of its row's largest, and the dropped digit
pairs weigh below 2^-55 of the product of the two row maxima, so the sum of K terms is
within K 2^-54 max|a_i| max|b_j|, plus the rounding of the result.  Factorizations: the
standard bounds, 4 n u sqrt(A_ii A_jj) for L L' - A and 8 n u cond(A) ||A^-1|| for the
inverse.
"""
import ctypes as C

import numpy as np
import pytest

from cosmicblup_gb300._lib import lib, ptr

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def gemm(handle, A, B, trans):
    m, k = A.shape
    n = B.shape[1] if trans else B.shape[0]
    out = np.empty((m, n))
    handle.check(lib().cbx_selftest_fx64_gemm(handle.raw, ptr(A), ptr(B), m, n, k, 1 if trans else 0, 0, ptr(out), None))
    return out


def chol(handle, A, inverse):
    n = A.shape[0]
    out = np.full((n, n), np.nan)
    ld, ok = C.c_double(0), C.c_int32(0)
    handle.check(lib().cbx_selftest_fx64_chol(handle.raw, ptr(A), n, 1 if inverse else 0, 0, ptr(out), C.byref(ld),
                                              C.byref(ok), None))
    return out, ld.value, ok.value


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (128, 64, 32), (129, 65, 33), (127, 63, 128), (40, 200, 129), (260, 130, 700)])
@pytest.mark.parametrize("trans", [False, True])
def test_product_edges(handle, m, n, k, trans):
    rng = np.random.default_rng(m + 10 * n + 100 * k)
    # rows of very different size, and large and small entries within a row
    A = rng.standard_normal((m, k)) * 10.0 ** rng.integers(-8, 9, (m, 1)) * 10.0 ** rng.integers(-3, 1, (m, k))
    B = rng.standard_normal((n, k)) * 10.0 ** rng.integers(-8, 9, (n, 1))
    A[m // 2, :] = 0.0
    out = gemm(handle, A, np.ascontiguousarray(B.T) if trans else B, trans)
    ref = A.astype(np.longdouble) @ B.T.astype(np.longdouble)
    tol = k * 2.0 ** -54 * np.abs(A).max(1)[:, None] * np.abs(B).max(1)[None, :] + 2 * U * np.abs(ref)
    assert (np.abs(out - ref) <= tol).all()


def test_product_of_non_finite_rows(handle):
    A = np.ones((130, 40))
    A[3, 7], A[129, 0] = np.nan, np.inf
    out = gemm(handle, A, np.ones((70, 40)), False)
    bad = np.zeros(130, bool)
    bad[[3, 129]] = True
    assert not np.isfinite(out[bad]).any() and (out[~bad] == 40.0).all()


def spd(n, rng):
    X = rng.standard_normal((n, n + 8))
    d = 10.0 ** rng.uniform(-2, 2, n)          # unequal scales, as the rows of an MME
    A = (X @ X.T / n + 0.3 * np.eye(n)) * d[:, None] * d[None, :]
    return 0.5 * (A + A.T), d


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 257, 640, 3100])
def test_factor_and_inverse(handle, n):
    A, d = spd(n, np.random.default_rng(n))
    L, ld, ok = chol(handle, A, False)          # column-major upper = row-major lower
    assert ok and (np.triu(L, 1) == 0).all()
    sc = np.sqrt(np.diag(A))
    assert (np.abs(L @ L.T - A) <= 4 * n * U * sc[:, None] * sc[None, :] + 8 * n * U).all()
    ref = np.linalg.slogdet(A)[1]
    assert abs(ld - ref) <= 1e-12 * max(1.0, np.abs(np.log(np.diag(L))).sum() * 2)
    Ai, ld2, ok = chol(handle, A, True)
    assert ok and abs(ld2 - ld) <= 1e-12 * max(1.0, abs(ld)) and (Ai == Ai.T).all()
    # scaled by the diagonal, where the condition of the problem is that of the scaled matrix
    As, Is = A / d[:, None] / d[None, :], Ai * d[:, None] * d[None, :]
    w = np.linalg.eigvalsh(As)
    assert np.abs(Is - np.linalg.inv(As)).max() <= 8 * n * U * w[-1] / w[0] / w[0]


def test_not_positive_definite(handle):
    for n, i in ((5, 4), (40, 33), (300, 299), (300, 0)):
        A = np.eye(n)
        A[i, i] = -1e-3
        assert chol(handle, A, False)[2] == 0
        assert chol(handle, A, True)[2] == 0
    A = np.eye(70)
    A[60, 2] = A[2, 60] = np.nan
    assert chol(handle, A, True)[2] == 0
