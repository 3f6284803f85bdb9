"""The one-null-direction path of the eigen-bending inverse (reml.cu, deflate_ones) as a
numpy model of its steps, against the oracle's invert_psd_matrix (CPU, oracle only).

One inverse N = (M + c v v')^-1, v = 1/sqrt(n), bounds the second eigenvalue from below;
the smallest eigenvalue's vector comes from u <- N (rho u + c (v'u) v), and the inverse off
it from N and two rank-1 terms.  The steps multiply an error by |rho| / lambda_i: the path
is left when |rho| is not far below lambda_2, as it is for clearly negative rho.
"""
import numpy as np
import pytest

from cosmicblup_gb300.synth import simulate_bed
from oracle.grm import vanraden_grm
from oracle.mme import invert_psd_matrix

EPS = 1e-6
U = 2.0 ** -53


def positive_definite(A):
    try:
        np.linalg.cholesky(A)
    except np.linalg.LinAlgError:
        return False
    return True


def deflate_ones(M):
    """The device path's steps; None where it leaves the matrix to the other paths."""
    n = M.shape[0]
    v = np.full(n, 1.0 / np.sqrt(n))
    c = np.abs(M).sum(axis=0).max()
    if not v @ M @ v < EPS:
        return None
    T = M + c * np.outer(v, v)
    if not positive_definite(T):
        return None
    N = np.linalg.inv(T)
    bound = np.abs(N).sum(axis=0).max()
    if not bound < 0.99 / (100 * EPS):
        if not positive_definite(T - 100 * EPS * np.eye(n)):
            return None
        bound = 1.0 / (100 * EPS)
    u, rho = v.copy(), 0.0
    for it in range(32):
        u = N @ (rho * u + c * (v @ u) * v)
        u /= np.linalg.norm(u)
        rho = u @ M @ u
        q = abs(rho) * bound
        if not q < 0.25:
            return None
        if it > 0 and q ** (it + 1) < 1e-16:
            break
    if not rho < EPS or not np.linalg.norm(M @ u - rho * u) <= 32 * n * U * c:
        return None
    w = N @ u
    uw = u @ w
    a = w - uw * u
    return (N - np.outer(u, w) - np.outer(w, u) + (uw + 1 / EPS) * np.outer(u, u)
            + rho / (1 - rho * uw) * np.outer(a, a))


@pytest.mark.parametrize("n,m,taken,seed", [(300, 2000, True, 1000), (500, 4000, True, 1001), (400, 300, False, 1002)])
def test_relationship_matrices(n, m, taken, seed):
    bed, _ = simulate_bed(n, m, seed=seed, p_lo=0.05, miss=0.01)
    G = vanraden_grm(bed, n, m)["G"]
    for a in (0.0, 1e-7, 3e-6):
        got = deflate_ones(G - a)
        assert (got is not None) == taken
        if taken:
            ref = invert_psd_matrix(G - a)
            assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()
    for a in (1e-4, 0.01, 0.05, 0.2):
        assert deflate_ones(G - a) is None


@pytest.mark.parametrize("lo,rho", [(1e-3, -1e-2), (1e-2, -0.1), (0.05, -0.5), (1e-2, -1e-2), (1e-3, -1e-7),
                                    (2e-4, 5e-7), (0.5, -1e-3)])
@pytest.mark.parametrize("tilt", [0.0, 0.03])
def test_never_a_wrong_inverse(lo, rho, tilt):
    n = 300
    rng = np.random.default_rng(17)
    B = rng.standard_normal((n, n))
    B[:, 0] = 1.0 + tilt * rng.standard_normal(n)
    Q, _ = np.linalg.qr(B)
    M = (Q * np.concatenate([[rho, lo], np.exp(rng.uniform(np.log(lo), np.log(2.0), n - 2))])) @ Q.T
    M = 0.5 * (M + M.T)
    got = deflate_ones(M)
    if rho <= -1e-2 or (tilt == 0.0 and rho < 0 and -rho >= 1e-2 * lo):
        assert got is None
    if got is not None:
        ref = invert_psd_matrix(M)
        assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()
    elif tilt == 0.0 and abs(rho) < EPS:
        assert False, "one eigenvalue within eps of zero along all-ones belongs to this path"
