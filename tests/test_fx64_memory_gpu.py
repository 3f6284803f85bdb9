"""What the digit factorizations need in memory, and their products by row groups where
the digits do not fit: the totals are the same integers, so the results have the same bits.
"""
import ctypes as C
import threading
import time

import numpy as np
import pytest

from cosmicblup_gb300 import Handle, invert_psd
from cosmicblup_gb300._lib import lib, ptr

pytestmark = pytest.mark.gpu


@pytest.fixture()
def limited():
    with Handle(0) as h:
        yield h, lambda b: h.check(lib().cbx_selftest_digit_limit(h.raw, b))


def inverse(h, A):
    n = A.shape[0]
    out = np.full((n, n), np.nan)
    ld, ok = C.c_double(0), C.c_int32(0)
    h.check(lib().cbx_selftest_fx64_chol(h.raw, ptr(A), n, 1, 0, ptr(out), C.byref(ld), C.byref(ok), None))
    assert ok.value
    return out


# the digits of one row tile of 128 take 64 KB for 32 columns; groups of one, two and three
# row tiles, the last group full or not
@pytest.mark.parametrize("n,tiles", [(1, 1), (128, 1), (129, 1), (300, 1), (640, 1), (640, 2), (700, 2), (700, 3), (1100, 2)])
def test_inverse_by_row_groups(limited, n, tiles):
    h, limit = limited
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, n + 4))
    A = X @ X.T / n + 0.1 * np.eye(n)
    whole = inverse(h, A)
    ks = (n + 127) // 128 * 4
    limit(tiles * ks * 65536)
    parts = inverse(h, A)
    assert np.array_equal(whole, parts)
    limit(1)                               # one row tile at least
    assert np.array_equal(whole, inverse(h, A))


def test_eigen_bending_inverse_by_row_groups(limited):
    h, limit = limited
    n = 600
    rng = np.random.default_rng(3)
    X = rng.standard_normal((n, 3 * n))
    X -= X.mean(0)
    G = X @ X.T / (3 * n)                  # one null direction, along all-ones
    whole = invert_psd(h, G)
    limit(2 * 20 * 65536)
    assert np.array_equal(whole, invert_psd(h, G))


def test_peak_of_the_eigen_bending_inverse(limited):
    """M, the result and the factorization's triangle: 24 n^2 bytes, and 8 n^2 of digits where
    the memory has them; with the digits in two groups of 2,048 rows, 4,096 x 16 bytes a column."""
    torch = pytest.importorskip("torch")
    h, limit = limited
    n = 10000
    g = torch.Generator().manual_seed(1)
    X = torch.randn(n, 600, generator=g, dtype=torch.float64)
    X -= X.mean(0)
    G = (X @ X.T).numpy() / 600
    G += 0.05 * (np.eye(n) - 1.0 / n)
    low, stop = [0], threading.Event()

    def poll():
        while not stop.is_set():
            low[0] = min(low[0], torch.cuda.mem_get_info()[0])
            time.sleep(2e-4)

    for lim, digits in ((0, 8.0 * n * n), (2048 * n * 16, 4096 * 16.0 * n)):
        limit(lim)
        invert_psd(h, G[:300, :300].copy(), download=False)      # library handles and code
        free = low[0] = torch.cuda.mem_get_info()[0]
        stop.clear()
        t = threading.Thread(target=poll)
        t.start()
        invert_psd(h, G, download=False)
        stop.set()
        t.join()
        # panels, diagonal blocks and a margin: 20 KB a row
        assert free - low[0] <= 24.0 * n * n + digits + 20480.0 * n
        invert_psd(h, G[:300, :300].copy(), download=False)
