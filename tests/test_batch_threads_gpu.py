"""Many handles solving at once on host threads, their PCG iterations captured and replayed as
graphs: a batch with 16 workers runs through, again and again, and gives what one worker gives."""
import numpy as np
import pytest

from cosmicblup_gb300 import BatchProblem, RemlConfig, batch_reml
from cosmicblup_gb300.mme import FP64, MIXED
from cosmicblup_gb300.synth import genetic_values, simulate_bed, simulate_gblup_records
from cosmicblup_gb300.vce import MODE_EM
from oracle.mme import build_fixed_design

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def problems():
    rng = np.random.default_rng(9)
    out = []
    for i in range(48):
        n, m = int(rng.integers(300, 1300)), int(rng.integers(1500, 3000))
        bed, _ = simulate_bed(n, m, seed=900 + i, p_lo=0.05, miss=0.01)
        g = genetic_values(bed, n, m, seed=950 + i, var_a=0.4)
        rec = simulate_gblup_records(n, 5, g, seed=990 + i, var_e=0.6)
        p, rows, _ = build_fixed_design(rec["cats"])
        out.append(BatchProblem(bed=bed, n=n, m=m, y=rec["y"], aid=rec["aid"], rows=rows, p=p))
    return out


@pytest.mark.parametrize("precision", [MIXED, FP64])
def test_sixteen_workers(problems, precision):
    cfg = RemlConfig.default(mode=MODE_EM, precision=precision, max_iter=3)
    one = batch_reml(problems, cfg, workers=1)
    for _ in range(4):
        many = batch_reml(problems, cfg, workers=16)
        for a, b in zip(one, many):
            assert b.status == 0 and a.iterations == b.iterations
            assert abs(a.var_u - b.var_u) <= 1e-12 * a.var_u and abs(a.var_e - b.var_e) <= 1e-12 * a.var_e
