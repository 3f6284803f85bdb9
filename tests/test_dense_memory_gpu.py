"""The dense AI step where the digits of its products do not fit the memory (row groups, the same
bits), and what a large one leaves on the handle: Z A Z' and the device copies of the MME,
no digits and no scratch."""
import numpy as np
import pytest

from cosmicblup_gb300 import AIREML, DeviceMME, Handle, RemlConfig
from cosmicblup_gb300._lib import lib
from cosmicblup_gb300.vce import MODE_DENSE

pytestmark = pytest.mark.gpu


def reml(h, n, Q, steps, seed=7, p=3):
    rng = np.random.default_rng(seed)
    lvl = rng.integers(0, p, n)
    y = 5.0 + lvl + rng.standard_normal(n)
    rows = [[(0, 1.0)] + ([(int(k), 1.0)] if k else []) for k in lvl]
    m = DeviceMME(h, y, np.arange(1, n + 1), rows, p, n)
    m.set_qinv_dense(Q)
    r = AIREML(m, 0.5, 0.8, RemlConfig.default(mode=MODE_DENSE, max_iter=steps, tol=0.0))
    r.solve()
    return r.var_u, r.var_e, r.history[-1]["logL"], np.array(r.solution)


@pytest.mark.parametrize("n,tiles", [(128, 1), (300, 1), (300, 2), (515, 2)])
def test_dense_steps_by_row_groups(n, tiles):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 2 * n))
    Q = np.linalg.inv(X @ X.T / (2 * n) + 0.05 * np.eye(n))
    with Handle(0) as h:
        whole = reml(h, n, Q, 3)
        h.check(lib().cbx_selftest_digit_limit(h.raw, tiles * ((n + 31) // 32) * 65536))
        parts = reml(h, n, Q, 3)
    assert whole[:3] == parts[:3] and np.array_equal(whole[3], parts[3])


def test_a_large_step_leaves_no_scratch():
    torch = pytest.importorskip("torch")
    n = 8400
    Q = np.eye(n)
    Q += 0.01 / n
    with Handle(0) as h:
        y = np.random.default_rng(1).standard_normal(n)
        m = DeviceMME(h, y, np.arange(1, n + 1), [[(0, 1.0)]] * n, 1, n)
        m.set_qinv_dense(Q)
        r = AIREML(m, 0.5, 0.8, RemlConfig.default(mode=MODE_DENSE, max_iter=1, tol=0.0))
        free = torch.cuda.mem_get_info()[0]
        r.run_iteration()
        kept = free - torch.cuda.mem_get_info()[0]
    # Z A Z' and 256 MB for library handles and vectors
    assert kept <= 8 * n * n + (256 << 20)
