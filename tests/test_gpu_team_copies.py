"""Teams of one LP advance their scheduling fields in the warps' copies and write
them down at the next finisher or at the end of a launch.  The per-pass mode
(``persistent=False``) has no copies: a solve in either mode, cut into step
budgets that end inside runs of normal iterations, must give the same bits."""

import numpy as np
import pytest

from sovereign_moe_b200 import workloads
from sovereign_moe_b200.batch import BatchEngine
from sovereign_moe_b200.pdlp import PDLPParams

pytestmark = pytest.mark.gpu


def _lp(m, n, per_col, seed, long_rows=0):
    rng = np.random.default_rng(seed)
    cp, ci = workloads.random_structure(rng, m, np.minimum(per_col, m) * np.ones(n, dtype=np.int64))
    if long_rows:                 # the last column entry of most columns goes to one of a few rows
        ci = ci.copy()
        cols = np.repeat(np.arange(n), np.diff(cp))
        last = cp[1:] - 1
        rows = m + cols[last] % long_rows
        ci[last] = rows
        m += long_rows
    cx = rng.standard_normal(ci.shape[0])
    return workloads.known_optimum(rng, m, n, cp, ci.astype(np.int32), cx).problem


def _run(probs, params, persistent, budgets):
    with BatchEngine(max_slots=len(probs), persistent=persistent) as eng:
        slots = [eng.admit(p, params) for p in probs]
        k, active = 0, len(probs)
        while active:
            active = eng.step(budgets[k % len(budgets)])
            k += 1
        sols = [eng.fetch(s) for s in slots]
    return [(s.iterations, int(s.status), s.info.step_size, s.info.primal_weight, s.info.restarts,
             s.info.rejected_steps, tuple(map(tuple, s.info.history)), s.x.tobytes(),
             s.y.tobytes(), s.reduced_costs.tobytes()) for s in sols]


@pytest.mark.parametrize("check,every,limit", [(64, 8, 300), (64, 8, 203), (5, 3, 61), (10, 1, 40),
                                               (7, 64, 50), (64, 8, 8)])
@pytest.mark.parametrize("shape", [(3, 5, 2, 0), (230, 700, 6, 0), (60, 4000, 3, 2)])
def test_budgets_and_launch_modes_give_the_same_bits(shape, check, every, limit):
    m, n, per_col, long_rows = shape
    prob = _lp(m, n, per_col, 3, long_rows)
    params = PDLPParams(device="gpu", eps_abs=1e-6, eps_rel=1e-6, check_every=check,
                        stepsize_every=every, max_iter=limit)
    ref = _run([prob], params, False, [1 << 16])
    for budgets in ([1 << 16], [37], [1, 2, 3, 61]):
        assert _run([prob], params, True, budgets) == ref


def test_several_lps_in_teams_of_their_own():
    probs = [_lp(m, 3 * m + 1, 5, m, lr) for m, lr in ((4, 0), (70, 0), (500, 0), (40, 1), (900, 0))]
    params = PDLPParams(device="gpu", eps_abs=1e-6, eps_rel=1e-6, max_iter=700)
    ref = _run(probs, params, False, [1 << 16])
    assert _run(probs, params, True, [1 << 16]) == ref
    assert _run(probs, params, True, [101, 7]) == ref
