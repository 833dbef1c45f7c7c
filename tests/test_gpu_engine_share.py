"""A step's time, bytes, iterations and launches by engine: LPs on chip are not
counted as work of the block teams, whose bytes are the HBM roofline's."""

import numpy as np
import pytest

from sovereign_moe_b200 import workloads
from sovereign_moe_b200.batch import BatchEngine
from sovereign_moe_b200.pdlp import PDLPParams

pytestmark = pytest.mark.gpu

CHIP, TEAM = (63, 65, 5), (2300, 9100, 8)


def _lp(m, n, per_col):
    rng = np.random.default_rng([m, n])
    cp, ci = workloads.random_structure(rng, m, np.full(n, per_col))
    return workloads.known_optimum(rng, m, n, cp, ci, rng.standard_normal(ci.shape[0])).problem


def _bytes(prob):
    m, n, nnz = int(prob.A.m), int(prob.A.n), int(prob.A.nnz)
    return 24.0 * nnz + 4 * (m + 1) + 4 * (n + 1) + 8 * (10.0 * m + 11.0 * n)


@pytest.mark.parametrize("shapes", [[CHIP], [TEAM], [CHIP, TEAM, CHIP]])
@pytest.mark.parametrize("persistent", [True, False])
def test_shares_add_up_and_each_engine_has_its_own(require_gpu, shapes, persistent):
    probs = [_lp(*s) for s in shapes]
    params = PDLPParams(device="gpu", eps_abs=0.0, eps_rel=0.0, max_iter=128)
    with BatchEngine(max_slots=len(probs), persistent=persistent) as eng:
        slots = [eng.admit(p, params) for p in probs]
        assert eng.step(200) == 0                   # fewer steps than move an LP off chip
        total, team, chip = eng.last_timing(), eng.last_engine(False), eng.last_engine(True)
        assert [eng.fetch(s).iterations for s in slots] == [128] * len(probs)
    on_chip = [s == CHIP and persistent for s in shapes]
    for share, mine in ((chip, on_chip), (team, [not c for c in on_chip])):
        ms, by, its, launches = share
        assert its == 128 * sum(mine)
        assert by == sum(128 * _bytes(p) for p, own in zip(probs, mine) if own)
        assert (ms > 0) == (launches > 0) == any(mine)
    assert total[2] == team[2] + chip[2]
    assert total[1] == pytest.approx(team[1] + chip[1])
    assert total[0] == pytest.approx(team[0] + chip[0], rel=1e-4)
