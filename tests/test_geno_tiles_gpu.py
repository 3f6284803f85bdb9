"""Genotype products at the edges of their tiles: 16 and 64 samples, 256 SNPs and samples,
2048 samples, 4096 SNPs.  Same oracle and bounds as test_geno_gpu.py."""
import numpy as np
import pytest

from cosmicblup_gb300 import DeviceGenotypes
from oracle.geno import compute_stats, multiply_z_v, multiply_zt_v

from test_geno_gpu import case, z_tol, zt_tol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [
    (15, 31), (16, 32), (17, 33), (63, 255), (64, 256), (65, 257), (255, 16), (256, 15), (257, 17),
    (2047, 40), (2048, 64), (2049, 65), (40, 4095), (64, 4096), (33, 4097), (4097, 260), (300, 8300),
])
def test_tile_edges(handle, n, m):
    bed, g = case(n, m, seed=3 * n + m, miss=0.2)
    d = DeviceGenotypes(bed, n, m, handle)
    mean, inv = compute_stats(g)
    rng = np.random.default_rng(n + 5 * m)
    v, u = rng.standard_normal(n) * 10.0**rng.integers(-6, 3, n), rng.standard_normal(m)
    assert np.all(np.abs(d.multiply_Zt_v(v) - multiply_zt_v(g, mean, inv, v)) <= zt_tol(v[:, None], mean, inv)[:, 0])
    assert np.abs(d.multiply_Z_v(u) - multiply_z_v(g, mean, inv, u)).max() <= z_tol(u, mean, inv)
