"""The FP64 solver's block product where the digits of the block do not fit the memory: the
CUDA-core product takes its place, on the same solves as with digits."""
import numpy as np
import pytest

from cosmicblup_gb300 import DeviceMME, Handle
from cosmicblup_gb300._lib import lib
from cosmicblup_gb300.mme import FP64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(900, 12), (1100, 40), (1000, 64), (900, 70)])
def test_solves_without_digits(n, k):
    rng = np.random.default_rng(n + k)
    X = rng.standard_normal((n, n + 20))
    Q = np.linalg.inv(X @ X.T / n + 0.1 * np.eye(n)) + 3.0
    Q = 0.5 * (Q + Q.T)
    B = rng.standard_normal((n + 1, k))
    V = rng.standard_normal((n, k))
    L = np.zeros((n + 1, n + 1))
    L[0, 0] = n
    L[0, 1:] = L[1:, 0] = 1.0
    L[1:, 1:] = np.eye(n) + 1.3 * Q
    ref = np.linalg.solve(L, B)
    bound = np.linalg.cond(L) * 1e-11 * np.linalg.norm(B, axis=0).max()
    with Handle(0) as h:
        for limit in (0, 1, 0):
            h.check(lib().cbx_selftest_digit_limit(h.raw, limit))
            m = DeviceMME(h, rng.standard_normal(n) + 4, np.arange(1, n + 1), [[(0, 1.0)]] * n, 1, n)
            m.set_qinv_dense(Q)
            got, it, rel = m.pcg_solve(1.3, B, tol=1e-12, precision=FP64)
            assert (rel < 1e-12).all()
            assert np.linalg.norm(got - ref, axis=0).max() <= bound / np.abs(np.linalg.eigvalsh(L)).max()
            qv = Q.astype(np.longdouble) @ V
            assert (np.abs(m.qinv_apply(V) - qv) <= n * 2.0 ** -50 * (np.abs(Q) @ np.abs(V))).all()
