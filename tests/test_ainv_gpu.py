"""A^-1 by generations on several host threads against the oracle's sequential scan:
pedigrees with and without enough animals for a second thread, single parents, and one
that lists parents after their progeny (the sequential scan's case).

The same operations in the same order, but for the multiply-adds that the host compiler
contracts: each of an animal's at most n terms of F (below 2) then differs by a rounding,
so F and the Mendelian variance dii are within t = n 2^-51, 1 / dii within t / dii of itself,
and A^-1's entries, sums of multiples of 1 / dii of at most the largest diagonal in
magnitude, within t / min dii of that."""
import numpy as np
import pytest

from cosmicblup_gb300 import ainv_henderson
from oracle.ped import ainv_henderson as o_ainv

pytestmark = pytest.mark.gpu


def same(handle, dam, sire):
    got = ainv_henderson(handle, dam, sire, with_inbreeding=True)
    want = o_ainv(dam, sire)
    tol = dam.size * 2.0 ** -51
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert np.abs(got[3] - want[3]).max() <= tol and np.abs(got[4] - want[4]).max() <= tol
    assert np.abs(got[2] - want[2]).max() <= tol / want[4].min() * np.abs(want[2]).max()


@pytest.mark.parametrize("n,back", [(1, 1), (255, 40), (1500, 60), (3000, 2999)])
def test_ordered_pedigree(handle, n, back):
    rng = np.random.default_rng(n)
    i = np.arange(n)
    dam = np.where(i > 0, i - 1 - rng.integers(0, np.minimum(np.maximum(i, 1), back)), -1)
    sire = np.where(i > 0, i - 1 - rng.integers(0, np.minimum(np.maximum(i, 1), back)), -1)
    dam[rng.random(n) < 0.2] = -1
    sire[rng.random(n) < 0.2] = -1
    same(handle, dam, sire)


def test_progeny_before_parents(handle):
    rng = np.random.default_rng(5)
    n = 400
    perm = rng.permutation(n)
    dam, sire = np.full(n, -1), np.full(n, -1)
    for k in range(1, n):
        dam[perm[k]] = perm[rng.integers(0, k)]
        sire[perm[k]] = perm[rng.integers(0, k)]
    # the scan leaves coefficients behind here, as the reference's does, and dii can come
    # close to 0, so values are not settled to a bound: the pattern of A^-1 is
    got, want = ainv_henderson(handle, dam, sire, with_inbreeding=True), o_ainv(dam, sire)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    founders = (dam < 0) & (sire < 0)
    assert (got[3][founders] == 0.0).all() and (got[4][founders] == 1.0).all()
