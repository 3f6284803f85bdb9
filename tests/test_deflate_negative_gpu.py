"""Eigen-bending inverses of matrices whose eigenvalue along (or near) the all-ones
direction is negative: a relationship matrix from which a constant was taken, and spectra
with one negative eigenvalue whose vector is tilted off all-ones.  The one-null-direction
path's steps amplify an error there unless |rho| is far below the next eigenvalue.

Bound: eps = 1e-6 replaces the negative eigenvalue in sums with terms of the size of
||M||, each rounded at 2^-53, and the result's largest entries are 1 / eps times the
eigenvector's products; hence 4 2^-53 ||M|| / eps of the largest entry, and 1e-9 (the
parity bar of the inverse) where that is less.
"""
import numpy as np
import pytest

from cosmicblup_gb300 import invert_psd
from cosmicblup_gb300.synth import simulate_bed
from oracle.grm import vanraden_grm
from oracle.mme import invert_psd_matrix

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
EPS = 1e-6


def check(handle, M, ridge=0.0):
    got = invert_psd(handle, M, ridge=ridge)
    ref = invert_psd_matrix(M, ridge)
    bound = max(1e-9, 4 * U * np.linalg.norm(M, 2) / EPS)
    assert (got == got.T).all()
    assert np.abs(got - ref).max() <= bound * np.abs(ref).max()


@pytest.fixture(scope="module", params=[(300, 2000), (1000, 8000)], ids=["n300", "n1000"])
def grm(request):
    n, m = request.param
    bed, _ = simulate_bed(n, m, seed=1000, p_lo=0.05, miss=0.01)
    return vanraden_grm(bed, n, m)["G"]


@pytest.mark.parametrize("a", [0.0, 1e-6, 1e-4, 0.01, 0.05, 0.2])
def test_constant_taken_from_a_grm(handle, grm, a):
    check(handle, grm - a)


@pytest.mark.parametrize("lo,rho", [(1e-3, -1e-2), (1e-2, -0.1), (0.05, -0.5), (1e-2, -1e-2), (1e-3, -1e-5),
                                    (1e-3, -1e-7), (2e-4, 5e-7), (0.5, -1e-3)])
@pytest.mark.parametrize("tilt", [0.0, 0.03])
def test_one_negative_eigenvalue_near_all_ones(handle, lo, rho, tilt):
    n = 300
    rng = np.random.default_rng(17)
    q = np.full(n, 1.0) + tilt * rng.standard_normal(n)
    B = rng.standard_normal((n, n))
    B[:, 0] = q
    Q, _ = np.linalg.qr(B)
    ev = np.concatenate([[rho, lo], np.exp(rng.uniform(np.log(lo), np.log(2.0), n - 2))])
    M = (Q * ev) @ Q.T
    check(handle, 0.5 * (M + M.T))
