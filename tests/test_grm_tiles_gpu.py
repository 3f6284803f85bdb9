"""cbx_grm_bed at the edges of its tiles, chunks and parts.

Counts bit-exact; G within the stated bound n_valid 2^-46 / sum2pq + 4 ulp of the
exactly rounded one.
"""
import numpy as np
import pytest

from cosmicblup_gb300 import GrmBuilder, GrmOptions, PlinkReader
from cosmicblup_gb300.synth import encode_bed, simulate_bed
from oracle.grm import vanraden_grm_exact, xx_counts_valid

pytestmark = pytest.mark.gpu


def check(handle, bed, n, m):
    b = GrmBuilder(GrmOptions(), handle=handle)
    b.compute(PlinkReader.from_bytes(bed, n, m), keep_xx_counts=True)
    ex = vanraden_grm_exact(bed, n, m)
    np.testing.assert_array_equal(b.getXXCounts(), xx_counts_valid(bed, n, m))
    G = b.getGrm()
    bound = ex["n_valid"] * 2.0**-46 / ex["sum2pq"] + 4 * np.spacing(np.abs(ex["G"]))
    assert np.all(np.abs(G - ex["G"]) <= bound)
    assert np.array_equal(G, G.T)


@pytest.mark.parametrize("n,m", [
    (2, 3), (31, 64), (32, 65), (33, 63), (127, 129), (128, 640), (129, 1000),  # tile and step edges
    (33, 8200), (40, 17000),     # 8192-SNP chunks, in parts
    (8, 70000),                  # more SNPs than an int64 sum of e_j holds
    (385, 70), (1100, 700),      # items that fill the SMs once and more, uneven parts
])
def test_grm_edges(handle, n, m):
    check(handle, simulate_bed(n, m, seed=n + m, p_lo=0.02, miss=0.03)[0], n, m)


def test_grm_largest_digits(handle):
    """One allele count in all SNPs, that with the largest base-2048 digits of its mean:
    the chunks end where the sum of digits does, not at 8192 SNPs."""
    n, m = 257, 9000
    best = None
    for c in range(20, 2 * n - 20):
        a = int(float(np.float32(c / n)) * 2**29)
        d0 = (a + 1024) % 2048 - 1024
        d1 = ((a - d0 >> 11) + 1024) % 2048 - 1024
        best = max(best or (0, 0), (min(abs(d0), abs(d1)), c))
    assert best[0] > 700  # 4 * 700 * 8192 > 2^24
    rng = np.random.default_rng(5)
    g = np.zeros((m, n), np.int8)
    for j in range(m):
        g[j] = np.bincount(rng.permutation(2 * n)[:best[1]] // 2, minlength=n)
    check(handle, encode_bed(g), n, m)


def test_grm_copied_behind_the_tiles(handle):
    """Pinned output of an order whose copy follows the groups of tiles, against the copy
    of the whole matrix that pageable output gets: every entry, counts too."""
    import ctypes as C

    import torch

    from cosmicblup_gb300._lib import lib, ptr
    n, m = 7001, 130
    bed = np.frombuffer(simulate_bed(n, m, seed=8, miss=0.02)[0], np.uint8)
    out = []
    for pinned in (False, True):
        G = torch.full((n, n), float("nan"), dtype=torch.float64, pin_memory=pinned).numpy()
        s, k = C.c_double(), C.c_int64()
        handle.check(lib().cbx_grm_bed(handle.raw, ptr(bed), bed.size, n, m, C.c_float(0.01), 1, 2048, ptr(G), None,
                                       None, C.byref(s), C.byref(k)))
        out.append(G)
    np.testing.assert_array_equal(out[0], out[1])
    assert np.array_equal(out[1], out[1].T)
