"""The digit factorization (fx64.cu) of matrices with ill-conditioned pivot pairs: an
eigen-bent G^-1 holds 1e6 / n in every entry, and adjacent animals can be near-duplicates.

Bounds, as for any backward stable Cholesky: L L' - A within 4 n u sqrt(A_ii A_jj); the
inverse against one refined in extended precision within 1e-11 of its largest entry for
the eigen-bent matrices (LAPACK: up to 8e-12 at n = 64), and within eight times LAPACK's
own error for the near-duplicates; log-determinants within n u cond of the scaled matrix,
whose half is lost at most; a multi-trait solve within 5e-11 of the largest value.
"""
import ctypes as C

import numpy as np
import pytest

from cosmicblup_gb300 import solve_multi_trait
from cosmicblup_gb300._lib import lib, ptr
from cosmicblup_gb300.synth import simulate_bed
from oracle.grm import vanraden_grm
from oracle.mme import invert_psd_matrix
from oracle.mt import mt_lhs_rhs

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
LD = np.longdouble


def chol(handle, A, inverse):
    n = A.shape[0]
    out = np.full((n, n), np.nan)
    ld, ok = C.c_double(0), C.c_int32(0)
    handle.check(lib().cbx_selftest_fx64_chol(handle.raw, ptr(A), n, 1 if inverse else 0, 0, ptr(out), C.byref(ld),
                                              C.byref(ok), None))
    assert ok.value
    return out, ld.value


def product(A, X):
    """A X in extended precision: 20-bit slices, whose products are exact in FP64 sums."""
    def slices(M, axis):
        s = 2.0 ** np.ceil(np.log2(np.abs(M).max(axis=axis, keepdims=True)))
        M = M / s
        hi = np.rint(M * 2.0 ** 20) / 2.0 ** 20
        mid = np.rint((M - hi) * 2.0 ** 40) / 2.0 ** 40
        return s, (hi, mid, M - hi - mid)
    sa, a = slices(A, 1)
    sx, x = slices(X, 0)
    t = np.zeros((A.shape[0], X.shape[1]), LD)
    for w in (4, 3, 2, 1, 0):
        for i in range(3):
            if 0 <= w - i < 3:
                t += (a[i] @ x[w - i]).astype(LD)
    return t * sa.astype(LD) * sx.astype(LD)


def refined_inverse(A):
    X = np.linalg.inv(A)
    for _ in range(2):
        R = (np.eye(len(A)) - product(A, X)).astype(np.float64)
        X = X + X @ R
    return X


def bent(n, m):
    bed, _ = simulate_bed(n, m, seed=3, p_lo=0.05, miss=0.01)
    Q = invert_psd_matrix(vanraden_grm(bed, n, m)["G"])
    return 0.5 * (Q + Q.T)


def duplicates(n, delta):
    rng = np.random.default_rng(n)
    B = rng.standard_normal((n, n + 8))
    B[1::2] = B[0:n - 1:2] + delta * rng.standard_normal((n // 2, n + 8))
    return B @ B.T / n


MATRICES = [("bent", 64, 1000), ("bent", 301, 2500), ("bent", 700, 6000), ("bent", 1100, 9000),
            ("dup", 33, 1e-3), ("dup", 96, 1e-3), ("dup", 160, 1e-5), ("dup", 400, 1e-4)]


@pytest.mark.parametrize("kind,n,arg", MATRICES)
def test_ill_conditioned_pivot_pairs(handle, kind, n, arg):
    A = bent(n, arg) if kind == "bent" else duplicates(n, arg)
    L, ld = chol(handle, A, False)
    sc = np.sqrt(np.diag(A))
    assert (np.abs((product(L, np.ascontiguousarray(L.T)) - A).astype(np.float64)) <= 4 * n * U * np.outer(sc, sc)).all()
    w = np.linalg.eigvalsh(A / np.outer(sc, sc))
    Lr = np.linalg.cholesky(A)
    assert abs(ld - 2 * np.log(np.diag(Lr)).sum()) <= n * U * w[-1] / w[0]
    Ai, ld2 = chol(handle, A, True)
    assert (Ai == Ai.T).all() and abs(ld2 - ld) <= n * U * w[-1] / w[0]
    ref = refined_inverse(A)
    err = np.abs(Ai - ref).max() / np.abs(ref).max()
    Li = np.linalg.inv(Lr)
    lapack = np.abs(Li.T @ Li - ref).max() / np.abs(ref).max()
    assert err <= (1e-11 if kind == "bent" else 8 * lapack), (err, lapack)


def test_multi_trait_solve(handle):
    n, t = 300, 2
    Gi = bent(n, 2500)
    rng = np.random.default_rng(5)
    Vg, Ve = np.array([[0.3, 0.1], [0.1, 0.4]]), np.array([[0.7, 0.2], [0.2, 0.6]])
    Y, X = rng.standard_normal((n, t)) + 2.0, np.ones((n, 1))
    K, r, pt = mt_lhs_rhs(Y, X, Gi, Vg, Ve)
    x = np.linalg.solve(K, r)
    for _ in range(3):
        x = x + np.linalg.solve(K, (r - product(K, x[:, None])[:, 0]).astype(np.float64))
    s = solve_multi_trait(handle, Y, X, Vg, Ve, Ginv=Gi)
    assert np.abs(s["u"] - x[pt:]).max() <= 5e-11 * np.abs(x[pt:]).max()
    assert np.abs(s["beta"] - x[:pt]).max() <= 5e-11 * np.abs(x).max()
