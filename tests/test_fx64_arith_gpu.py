"""The kernels' own arithmetic against exact values: the reciprocal (the hardware's 20 bits,
one third-order step: e^3 < 2^-56 and two roundings, within 2^-52), the conversion of
the digit products' integer totals (nearest, so within half a unit in the last place), and a
product long enough for the totals to pass 2^63 on the way (432 chunks of 128), of
integers, whose sums are exact.
"""
from fractions import Fraction

import numpy as np
import pytest

from cosmicblup_gb300._lib import lib, ptr

pytestmark = pytest.mark.gpu


def test_reciprocal(handle):
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(1, 2, 200000) * 2.0 ** rng.integers(-900, 900, 200000),
                        2.0 ** np.arange(-1000, 1000), np.nextafter(2.0 ** np.arange(-900, 900), 0)])
    x[::3] *= -1
    y = np.empty_like(x)
    handle.check(lib().cbx_selftest_reciprocal(handle.raw, ptr(x), x.size, ptr(y)))
    one = np.longdouble(1)
    assert np.abs((y.astype(np.longdouble) * x - one)).max() <= 2.0 ** -52


def test_totals(handle):
    rng = np.random.default_rng(2)
    n = 6000
    bits = rng.integers(0, 62, (2, n))
    hi = (rng.integers(0, 2 ** 62, n) >> (62 - bits[0])) * rng.choice([-1, 1], n)
    lo = (rng.integers(0, 2 ** 62, n) >> (62 - bits[1])) * rng.choice([-1, 1], n)
    hi[:200] = 0                                             # 32 leading bits missing, and 64
    lo[100:200] = rng.integers(-9, 10, 100)
    lo[200:300] = 0
    k = np.arange(60)                                        # carries into the next power of two
    hi[300:360], lo[300:360] = (np.int64(1) << k), -1
    hi[360:420], lo[360:420] = -(np.int64(1) << k), 1
    hi[420:430], lo[420:430] = 0, 0
    hi[430:440], lo[430:440] = -1, 2 ** 32 + np.arange(10)   # small totals of large parts
    e = rng.integers(-890, 780, n).astype(np.int32)
    hi, lo = np.ascontiguousarray(hi, np.int64), np.ascontiguousarray(lo, np.int64)
    y = np.empty(n)
    handle.check(lib().cbx_selftest_from_totals(handle.raw, ptr(hi), ptr(lo), ptr(e), n, ptr(y)))
    for h, l, x, v in zip(hi.tolist(), lo.tolist(), e.tolist(), y.tolist()):
        exact = Fraction(h * 2 ** 32 + l) * Fraction(2) ** x
        assert 2 * abs(Fraction(v) - exact) <= Fraction(float(np.spacing(abs(v)))) if exact else v == 0.0


@pytest.mark.parametrize("k", [128 * 431, 128 * 432, 128 * 433 + 5])
def test_long_sums(handle, k):
    rng = np.random.default_rng(k)
    A = rng.integers(-2 ** 18, 2 ** 18, (70, k)).astype(np.float64)
    B = rng.integers(-2 ** 18, 2 ** 18, (33, k)).astype(np.float64)
    A[0], B[0] = 2.0 ** 18 - 1, 2.0 ** 18 - 1                 # the largest sum
    out = np.empty((70, 33))
    handle.check(lib().cbx_selftest_fx64_gemm(handle.raw, ptr(A), ptr(B), 70, 33, k, 0, 0, ptr(out), None))
    assert np.array_equal(out, (A.astype(np.int64) @ B.T.astype(np.int64)).astype(np.float64))
