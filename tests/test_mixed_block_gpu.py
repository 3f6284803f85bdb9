"""Mixed-precision solves of 32-, 64- and 128-wide blocks at orders around the 32-row tiles
of the gather, compared through the residual in extended precision (see
test_fp64_block_gpu.py): the refinement stops on the FP64 residual."""
import numpy as np
import pytest

from cosmicblup_gb300.mme import MIXED

from test_fp64_block_gpu import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [17, 33, 80])
@pytest.mark.parametrize("n", [31, 32, 33, 64, 65, 129])
def test_mixed_solves(handle, n, k):
    m, Q, rng = make(handle, n, 11 * n + k)
    B = rng.standard_normal((n + 1, k))
    lam = 1.3
    X, it, rel = m.pcg_solve(lam, B, tol=1e-10, precision=MIXED)
    L = np.zeros((n + 1, n + 1), dtype=np.longdouble)
    L[0, 0] = n
    L[0, 1:] = L[1:, 0] = 1.0
    L[1:, 1:] = np.eye(n) + lam * Q
    r = np.linalg.norm((B - L @ X).astype(float), axis=0) / np.linalg.norm(B, axis=0)
    # one rounding of A x in FP64 in the residual that the refinement stops on
    drift = 2.0 ** -50 * np.abs(L).sum(1).max() * np.linalg.norm(X, axis=0) / np.linalg.norm(B, axis=0)
    assert (rel < 1e-10).all() and (r <= 1e-10 + drift).all()
