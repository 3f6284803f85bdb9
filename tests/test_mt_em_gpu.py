"""The eigen-EM over several blocks against a plain restatement of its update, at sample
counts around one block (128) and past one wave of blocks, for one to eight traits.

Both make the same update from sums in another order; over the few iterations run each
entry of Vg and Ve is a sum of n terms of its own size, so they agree to n * 2^-50."""
import numpy as np
import pytest

from cosmicblup_gb300 import GrmBuilder, GrmOptions, MvEigenVce, MvOptions, PlinkReader, invert_psd
from cosmicblup_gb300.synth import simulate_bed

pytestmark = pytest.mark.gpu


def em(Y, X, G, iters):
    n, p = X.shape
    Q = np.linalg.qr(X, mode="complete")[0][:, p:]
    w, U = np.linalg.eigh(Q.T @ G @ Q)
    R = U.T @ Q.T @ Y
    w = np.maximum(w, 0.0)
    ne = n - p
    Vg = 0.5 * np.cov(Y.T, ddof=p + 1).reshape(Y.shape[1], -1) * (n - p - 1) / (ne - 1)
    Ve = Vg.copy()
    for _ in range(iters):
        P = np.linalg.inv(w[:, None, None] * Vg + Ve)
        q = np.einsum("iab,ib->ia", P, R)
        m = q[:, :, None] * q[:, None, :] - P
        d = np.where(w > 1e-12, w, 0.0)
        Vg, Ve = (Vg + Vg @ (d[:, None, None] * m).sum(0) @ Vg / ne, Ve + Ve @ m.sum(0) @ Ve / ne)
    return Vg, Ve


@pytest.mark.parametrize("n,t", [(60, 1), (130, 2), (131, 3), (400, 5), (700, 8), (1500, 3)])
def test_em_iterations(handle, n, t):
    rng = np.random.default_rng(10 * n + t)
    p = 2
    X = np.stack([np.ones(n), rng.integers(0, 2, n)], 1).astype(float)
    Z = rng.standard_normal((n, 2 * n))
    G = Z @ Z.T / (2 * n)
    Y = rng.standard_normal((n, t)) + np.linalg.cholesky(G + 0.01 * np.eye(n)) @ rng.standard_normal((n, t))
    v = MvEigenVce(handle, MvOptions(max_iter=4, tol=0.0))
    v.prepare(Y, X, G)
    v.runNullModel()
    Vg, Ve = em(Y, X, G, 4)
    tol = n * 2.0 ** -50
    assert v.iterations == 4
    assert np.abs(v.getVg() - Vg).max() <= tol * np.abs(Vg).max()
    assert np.abs(v.getVe() - Ve).max() <= tol * np.abs(Ve).max()


@pytest.mark.parametrize("n,t", [(129, 2), (320, 3), (513, 2)])
def test_g_recovered_from_the_device_inverse(handle, n, t):
    """Vg and Ve of the G that the handle's eigen-bent G^-1 stands for, against those of the
    bent G itself.  G^-1 has entries of 1 / (1e-6 n), each rounded at 2^-53 of that, and G's
    other eigenvalues are about 1: an error of 1e-16 * 1e6 / n * sqrt(n) a row, 1e-11 at
    these orders, and ten times that for the iterations' amplification."""
    m = 12 * n
    bed, _ = simulate_bed(n, m, seed=n, miss=0.02)
    b = GrmBuilder(GrmOptions(), handle=handle)
    b.compute(PlinkReader.from_bytes(bed, n, m))
    w, U = np.linalg.eigh(b.getGrm())
    G = (U * np.maximum(w, 1e-6)) @ U.T
    invert_psd(handle, None, n, download=False)
    rng = np.random.default_rng(n)
    X = np.stack([np.ones(n), rng.integers(0, 2, n)], 1).astype(float)
    Y = rng.standard_normal((n, t)) + np.linalg.cholesky(G + 0.01 * np.eye(n)) @ rng.standard_normal((n, t))
    out = []
    for g in (None, G):
        v = MvEigenVce(handle, MvOptions())
        v.prepare(Y, X, g)
        v.runNullModel()
        out.append((v.getVg(), v.getVe(), v.iterations))
    assert out[0][2] == out[1][2]
    for a, e in zip(out[0][:2], out[1][:2]):
        assert np.linalg.norm(a - e) <= 1e-10 * np.linalg.norm(e)
