"""The dense AI step's state belongs to one Qinv: a second MME of the same shape on the
same handle, with other records and another Qinv, gives what a new handle gives, and one
call per iteration gives what one call for all of them gives."""
import numpy as np
import pytest

from cosmicblup_gb300 import AIREML, DeviceMME, Handle, RemlConfig
from cosmicblup_gb300.vce import MODE_DENSE

pytestmark = pytest.mark.gpu


def problem(seed, n=150, p=3):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, 2 * n))
    G = X @ X.T / (2 * n) + 0.05 * np.eye(n)
    lvl = rng.integers(0, p, n)
    y = 5.0 + lvl + np.linalg.cholesky(G) @ rng.standard_normal(n) * 0.7 + rng.standard_normal(n)
    rows = [[(0, 1.0)] + ([(int(k), 1.0)] if k else []) for k in lvl]
    return y, np.arange(1, n + 1), rows, p, np.linalg.inv(G)


def run(h, pb, steps):
    y, aid, rows, p, Q = pb
    m = DeviceMME(h, y, aid, rows, p, y.size)
    m.set_qinv_dense(Q)
    r = AIREML(m, 0.5, 0.5, RemlConfig.default(mode=MODE_DENSE, max_iter=steps, tol=0.0))
    if steps == 3:
        r.solve()
        return r.var_u, r.var_e, r.history[-1]["logL"], r.solution
    for _ in range(3):
        r.run_iteration()
    return r.var_u, r.var_e, r.history[-1]["logL"], None


def test_second_mme_of_the_same_shape():
    a, b = problem(1), problem(2)
    with Handle(0) as h:
        run(h, a, 3)
        second = run(h, b, 3)
    with Handle(0) as h:
        fresh = run(h, b, 3)
        single = run(h, b, 1)
    assert second[:3] == fresh[:3] and np.array_equal(second[3], fresh[3])
    assert single[:3] == fresh[:3]
