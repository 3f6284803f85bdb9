"""Dense exact AI-REML and the recovered G of the multi-trait path with an eigen-bent G^-1
(1e6 / n in every entry), at orders where the factorization is one, two and many panels.

Reference: V = vu A + ve I and P from it, which are well conditioned (A = the eigen-bent
G), so FP64 gives them to about 1e-14.  Bounds: 4e-8 / n of the variances, four times what
LAPACK's Cholesky of Q = A^-1 leaves (1.1e-10 at n = 96, 3.8e-11 at 301), and 1e-9 of logL;
the recovered G's
variances within 1e-9 of those of A itself, where the EM's stopping rule at 1e-7 of them allows it.
"""
import numpy as np
import pytest

from cosmicblup_gb300 import AIREML, DeviceMME, MvEigenVce, MvOptions, RemlConfig, invert_psd
from cosmicblup_gb300.synth import genetic_values, simulate_bed, simulate_gblup_records
from cosmicblup_gb300.vce import MODE_DENSE
from oracle.grm import vanraden_grm
from oracle.mme import build_fixed_design

pytestmark = pytest.mark.gpu


def bent_pair(G):
    """The eigen-bent G and its inverse."""
    w, U = np.linalg.eigh(G)
    w = np.maximum(w, 1e-6)
    return (U * w) @ U.T, (U / w) @ U.T


def ai_step(y, X, A, vu, ve):
    """One AI step from (vu, ve) without halvings, and logL there."""
    n = y.size
    Vi = np.linalg.inv(vu * A + ve * np.eye(n))
    XVX = X.T @ Vi @ X
    P = Vi - Vi @ X @ np.linalg.solve(XVX, X.T @ Vi)
    Py = P @ y
    M = P @ A
    AI = 0.5 * np.array([[np.sum(M * M.T), np.sum(M * P)], [np.sum(M * P), np.sum(P * P)]])
    g = 0.5 * np.array([Py @ A @ Py - np.trace(M), Py @ Py - np.trace(P)])
    logL = lambda a, b: (lambda V: -0.5 * (np.linalg.slogdet(V)[1] + np.linalg.slogdet(X.T @ np.linalg.solve(V, X))[1]
                                           + y @ np.linalg.solve(V, y - X @ np.linalg.solve(
                                               X.T @ np.linalg.solve(V, X), X.T @ np.linalg.solve(V, y)))))(
                                                   a * A + b * np.eye(n))
    d = np.linalg.solve(AI, g)
    cur = logL(vu, ve)
    for _ in range(6):
        if vu + d[0] > 0 and ve + d[1] > 0 and logL(vu + d[0], ve + d[1]) > cur:
            break
        d = d / 2
    return vu + d[0], ve + d[1], logL(vu + d[0], ve + d[1])


@pytest.mark.parametrize("n,m", [(96, 1200), (301, 2500), (700, 6000), (1100, 9000)])
def test_dense_ai_step(handle, n, m):
    bed, _ = simulate_bed(n, m, seed=31, p_lo=0.05, miss=0.01)
    A, Q = bent_pair(vanraden_grm(bed, n, m)["G"])
    rec = simulate_gblup_records(n, 2, genetic_values(bed, n, m, seed=32, var_a=0.4), seed=33, var_e=0.6)
    p, rows, _ = build_fixed_design(rec["cats"])
    X = np.zeros((n, p))
    for i, r in enumerate(rows):
        for c, v in r:
            X[i, c] += v
    A = A[np.ix_(rec["aid"] - 1, rec["aid"] - 1)]
    dm = DeviceMME(handle, rec["y"], rec["aid"], rows, p, n)
    dm.set_qinv_dense(Q)
    r = AIREML(dm, 0.5, 0.5, RemlConfig.default(mode=MODE_DENSE, max_iter=1, tol=0.0))
    r.run_iteration()
    vu, ve, logL = ai_step(rec["y"], X, A, 0.5, 0.5)
    assert abs(r.var_u - vu) <= 4e-8 / n * vu and abs(r.var_e - ve) <= 4e-8 / n * ve
    assert abs(r.history[-1]["logL"] - logL) <= 1e-9 * abs(logL)


def test_recovered_g(handle):
    n, m = 320, 3000
    bed, _ = simulate_bed(n, m, seed=41, p_lo=0.05, miss=0.01)
    G = vanraden_grm(bed, n, m)["G"]
    A, _ = bent_pair(G)
    rng = np.random.default_rng(42)
    Y = np.linalg.cholesky(A) @ rng.standard_normal((n, 2)) + rng.standard_normal((n, 2)) + 1.0
    X = np.ones((n, 1))
    invert_psd(handle, G)
    out = []
    for g in (None, A):
        v = MvEigenVce(handle, MvOptions(max_iter=200, tol=1e-7))
        v.prepare(Y, X, g)
        v.runNullModel()
        out.append((v.iterations, v.getVg(), v.getVe()))
    assert out[0][0] == out[1][0]
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=0, atol=1e-9)
    np.testing.assert_allclose(out[0][2], out[1][2], rtol=0, atol=1e-9)
