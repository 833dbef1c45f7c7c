"""Teams of one LP: what a warp knows of its LP does not depend on when it reads it.

A warp that owns no tile of a pass does not hold up the pass's finisher, which
advances the LP's state.  The test hook makes such warps read 20 us late, after
a short pass has ended; every result must still be the per-pass mode's, bit for
bit: after checks with and without a restart, after the power iteration, after
line searches, with check periods that are no multiple of the step-size period,
and at launches that begin between any two of them.  (Under the hook no LP is
stepped on chip, so small LPs reach the teams too.)"""

import numpy as np
import pytest

from sovereign_moe_b200 import workloads
from sovereign_moe_b200.batch import BatchEngine
from sovereign_moe_b200.pdlp import PDLPParams

pytestmark = pytest.mark.gpu

LATE = 2


def _lp(m, n, per_col, seed=0):
    rng = np.random.default_rng([m, n, seed])
    cp, ci = workloads.random_structure(rng, m, np.full(n, min(per_col, m)))
    return workloads.known_optimum(rng, m, n, cp, ci, rng.standard_normal(ci.shape[0])).problem


def _dense_row(seed):
    """A row of more entries than a tile holds keeps an LP off chip."""
    rng = np.random.default_rng(seed)
    m, n = 3, 600
    ci = np.stack([np.zeros(n, dtype=np.int32), 1 + rng.integers(0, m - 1, n).astype(np.int32)], 1)
    return workloads.known_optimum(rng, m, n, np.arange(0, 2 * n + 1, 2), ci.reshape(-1),
                                   rng.standard_normal(2 * n)).problem


def _bits(probs, params, budgets=(1 << 16,), **cfg):
    with BatchEngine(max_slots=len(probs), **cfg) as eng:
        slots, codes = eng.admit_many(probs, params)
        assert codes == [0] * len(probs)
        k, active = 0, len(probs)
        while active:
            active = eng.step(budgets[k % len(budgets)])
            k += 1
        sols = [eng.fetch(s) for s in slots]
    return [(s.iterations, int(s.status), s.info.step_size, s.info.primal_weight, s.info.restarts,
             s.info.rejected_steps, tuple(map(tuple, s.info.history)), s.x.tobytes(),
             s.y.tobytes(), s.reduced_costs.tobytes()) for s in sols]


# one block (two of its four warps without tiles) to several; many more column
# tiles than row tiles (whole blocks without row tiles) and the reverse
SHAPES = [(3, 5, 2), (63, 65, 5), (230, 2025, 6), (40, 1700, 4), (1500, 300, 20)]


@pytest.mark.parametrize("check,every,limit", [(64, 8, 200), (5, 3, 61), (10, 4, 55), (7, 64, 50)])
@pytest.mark.parametrize("shape", SHAPES)
def test_late_reads_change_nothing(shape, check, every, limit):
    prob = _lp(*shape)
    params = PDLPParams(device="gpu", eps_abs=1e-6, eps_rel=1e-6, check_every=check,
                        stepsize_every=every, max_iter=limit)
    ref = _bits([prob], params, persistent=False)
    assert _bits([prob], params, test_withhold_arrival=LATE) == ref
    assert _bits([prob], params, budgets=(1, 2, 3, 29), test_withhold_arrival=LATE) == ref


def test_several_teams_of_one_lp_late_and_not():
    probs = [_lp(*s, seed=q) for q in range(4) for s in SHAPES] + [_dense_row(q) for q in range(4)]
    params = PDLPParams(device="gpu", eps_abs=1e-6, eps_rel=1e-6, max_iter=330)
    ref = _bits(probs, params, persistent=False)
    assert _bits(probs, params, test_withhold_arrival=LATE) == ref
    assert _bits(probs, params, budgets=(101, 7), test_withhold_arrival=LATE) == ref


def test_one_team_of_more_than_256_lps_beside_lps_on_chip():
    """More LPs than teams, none of which fits a cluster, and some on chip: one
    team steps the former by one budget, the latter stay on chip until 256
    teams are enough, in uneven step budgets."""
    big = [_dense_row(q) for q in range(5)]
    chip = [_lp(63, 65, 5), _lp(230, 2025, 6)]
    probs = [big[q % 5] for q in range(270)] + [chip[q % 2] for q in range(6)]
    params = PDLPParams(device="gpu", eps_abs=1e-6, eps_rel=1e-6, max_iter=700)
    ref_big = [_bits([p], params, persistent=False)[0] for p in big]
    ref_chip = [_bits([p], params, persistent=False)[0] for p in chip]
    ref = [ref_big[q % 5] for q in range(270)] + [ref_chip[q % 2] for q in range(6)]
    assert _bits(probs, params) == ref
    assert _bits(probs, params, budgets=(300, 1, 90)) == ref


def test_admission_between_steps_of_teams():
    """LPs that join teams of one LP between late steps equal themselves alone."""
    probs = [_lp(*s) for s in SHAPES]
    params = PDLPParams(device="gpu", eps_abs=1e-6, eps_rel=1e-6, max_iter=300)
    with BatchEngine(max_slots=len(probs), test_withhold_arrival=LATE) as eng:
        slots = []
        for p in probs:
            slots.append(eng.admit(p, params))
            eng.step(33)
        eng.run()
        got = [(s.iterations, s.x.tobytes(), s.y.tobytes()) for s in map(eng.fetch, slots)]
    ref = [_bits([p], params, persistent=False)[0] for p in probs]
    assert got == [(r[0], r[7], r[8]) for r in ref]
