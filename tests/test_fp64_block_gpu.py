"""The FP64 solver's block product on each of its paths -- one column, the CUDA-core product
and the digit product -- on both sides of the rule between the last two (ng^2 columns =
8e6), at column counts around 32 and 64 and at orders that leave a partial 128-row tile.

Q x is held to n 2^-50 of |Q||x|, which covers both products' bounds (an FP64 sum of n terms,
and K 2^-54 of the row maxima); solves stop on the residual, so they are compared through
it, computed in extended precision."""
import numpy as np
import pytest

from cosmicblup_gb300 import DeviceMME
from cosmicblup_gb300.mme import FP64

pytestmark = pytest.mark.gpu


def make(handle, n, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, n + 20))
    Q = np.linalg.inv(X @ X.T / n + 0.1 * np.eye(n)) + 3.0
    Q = 0.5 * (Q + Q.T)
    m = DeviceMME(handle, rng.standard_normal(n) + 4, np.arange(1, n + 1), [[(0, 1.0)]] * n, 1, n)
    m.set_qinv_dense(Q)
    return m, Q, rng


@pytest.mark.parametrize("n,k", [(130, 1), (130, 7), (500, 31), (500, 33), (897, 10), (899, 10), (1100, 32), (1280, 70)])
def test_qinv_product(handle, n, k):
    m, Q, rng = make(handle, n, n + k)
    X = rng.standard_normal((n, k)) * 10.0 ** rng.integers(-6, 7, k)
    ref = Q.astype(np.longdouble) @ X.astype(np.longdouble)
    assert (np.abs(m.qinv_apply(X) - ref) <= n * 2.0 ** -50 * (np.abs(Q) @ np.abs(X))).all()


@pytest.mark.parametrize("n,k", [(300, 1), (300, 3), (700, 12), (700, 20), (1100, 40), (900, 65)])
def test_fp64_solves(handle, n, k):
    m, Q, rng = make(handle, n, 7 * n + k)
    B = rng.standard_normal((n + 1, k))
    lam = 1.3
    X, it, rel = m.pcg_solve(lam, B, tol=1e-11, precision=FP64)
    L = np.zeros((n + 1, n + 1), dtype=np.longdouble)
    L[0, 0] = n
    L[0, 1:] = L[1:, 0] = 1.0
    L[1:, 1:] = np.eye(n) + lam * Q
    r = np.linalg.norm((B - L @ X).astype(float), axis=0) / np.linalg.norm(B, axis=0)
    # the recursive residual's drift: a rounding of A x per iteration
    drift = it.max() * 2.0 ** -50 * np.abs(L).sum(1).max() * np.linalg.norm(X, axis=0) / np.linalg.norm(B, axis=0)
    assert (rel < 1e-11).all() and (r <= 1e-11 + drift).all()
