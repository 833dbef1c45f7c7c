"""The resident engine (one LP per thread-block cluster, on chip) against the
per-pass engine, which shares none of its barriers, layouts or row loops.

Row sums, steps, tile partials and reduction trees are the same operations in
the same order in both, so every result must be the same bits: for LPs that
need clusters of 1 to 16 SMs and ones just beyond, with one and several lanes
per row, one and several reduction groups (64 tiles), in both precisions, alone
(clusters grow) and side by side, and cut into step budgets."""

import numpy as np
import pytest

from sovereign_moe_b200 import workloads
from sovereign_moe_b200.batch import BatchEngine
from sovereign_moe_b200.pdlp import PDLPParams

pytestmark = pytest.mark.gpu


def _lp(m, n, per_col, seed=0):
    rng = np.random.default_rng([m, n, seed])
    cp, ci = workloads.random_structure(rng, m, np.full(n, min(per_col, m)))
    return workloads.known_optimum(rng, m, n, cp, ci, rng.standard_normal(ci.shape[0])).problem


def _params(**kw):
    kw = {"device": "gpu", "eps_abs": 1e-6, "eps_rel": 1e-6, "max_iter": 330, **kw}
    return PDLPParams(**kw)


def _bits(probs, params, persistent, budgets=(1 << 16,), **cfg):
    with BatchEngine(max_slots=len(probs), persistent=persistent, **cfg) as eng:
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


# (rows, columns, entries per column): one tile; a ragged last tile; 53 entries
# per row (two lanes); 170 per row (four lanes); more than 64 column tiles; near
# the limits of 1, 2, 4, 8 and 16 SMs; beyond them (the team engine)
SHAPES = [(1, 1, 1), (2, 3, 2), (63, 65, 5), (64, 128, 5), (230, 2025, 6), (40, 1700, 4),
          (300, 4200, 5), (300, 900, 8), (500, 1500, 10), (700, 2800, 9), (900, 4500, 9),
          (1200, 6000, 9), (1400, 7000, 8), (2300, 9100, 8)]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", SHAPES)
def test_alone_equals_the_per_pass_engine(shape, precision):
    prob = _lp(*shape)
    params = _params(precision=precision)
    ref = _bits([prob], params, False)
    assert _bits([prob], params, True) == ref
    assert _bits([prob], params, True, budgets=(5, 33, 1, 64)) == ref


def test_side_by_side_in_every_cluster_size():
    probs = [_lp(*s, seed=q) for q in range(6) for s in SHAPES]
    params = _params(max_iter=150)
    assert _bits(probs, params, True) == _bits(probs, params, False)


@pytest.mark.parametrize("lanes", [1, 2, 8, 32])
def test_lanes(lanes):
    prob = _lp(120, 900, 7)
    params = _params(max_iter=100)
    assert _bits([prob], params, True, lanes_override=lanes) == \
        _bits([prob], params, False, lanes_override=lanes)


def test_line_search_failure_and_limits_inside_a_run():
    """A check period that is no multiple of the step-size period, an iteration
    limit inside a run of iterations, and one at its start."""
    prob = _lp(200, 600, 6)
    for kw in (dict(check_every=50, stepsize_every=7, max_iter=177),
               dict(check_every=64, stepsize_every=8, max_iter=64), dict(max_iter=1),
               dict(max_iter=0), dict(check_every=1, stepsize_every=1, max_iter=9),
               dict(check_every=1000, stepsize_every=3, max_iter=130)):
        params = _params(**kw)
        assert _bits([prob], params, True) == _bits([prob], params, False), kw


def test_cancel_and_retire_between_budgets():
    probs = [_lp(150, 500, 5, seed=q) for q in range(3)]
    with BatchEngine(max_slots=3) as eng:
        slots = [eng.admit(p, _params(max_iter=100_000, eps_abs=0.0, eps_rel=0.0)) for p in probs]
        assert eng.step(100) == 3
        eng.cancel(slots[1])
        eng.step(200)
        assert eng.done(slots[1]) and not eng.done(slots[0])
        eng.retire(slots[1])
        again = eng.admit(probs[1], _params())
        eng.cancel(slots[0])
        eng.cancel(slots[2])
        eng.run()
        got = eng.fetch(again)
    ref = _bits([probs[1]], _params(), False)[0]
    assert (got.iterations, got.x.tobytes()) == (ref[0], ref[7])


@pytest.mark.parametrize("order", [(0, 1, 2), (2, 1, 0)])
def test_engines_hand_over_to_each_other(order):
    """LPs that use up a whole launch on chip while another LP needs the team
    engine go on beside it there, and return on chip when it has finished."""
    lps = [(_lp(230, 2025, 6), _params(max_iter=4000, eps_abs=0.0, eps_rel=0.0)),
           (_lp(2300, 9100, 8), _params(max_iter=1500, eps_abs=0.0, eps_rel=0.0)),
           (_lp(40, 1700, 4), _params(max_iter=3000, eps_abs=0.0, eps_rel=0.0, precision="fp32"))]
    lps = [lps[i] for i in order]

    def run(group, budget):
        with BatchEngine(max_slots=len(group)) as eng:
            slots = [eng.admit(p, prm) for p, prm in group]
            while eng.step(budget):
                pass
            return [(s.iterations, s.info.restarts, s.x.tobytes(), s.y.tobytes())
                    for s in (eng.fetch(q) for q in slots)]

    alone = [run([lp], 1 << 30)[0] for lp in lps]
    assert run(lps, 1 << 30) == alone
    assert run(lps, 700) == alone


def test_more_lps_than_teams_take_turns():
    """Beyond 256 LPs the team engine steps its LPs by one budget, so LPs on chip
    stay there and take turns with it."""
    small, large = _lp(63, 65, 5), _lp(2300, 9100, 8)
    ps = _params(max_iter=500, eps_abs=0.0, eps_rel=0.0)
    pl = _params(max_iter=300, eps_abs=0.0, eps_rel=0.0)
    with BatchEngine(max_slots=270) as eng:
        slots = [eng.admit(small, ps) for _ in range(266)] + [eng.admit(large, pl) for _ in range(3)]
        while eng.step(400):
            pass
        got = [(s.iterations, s.x.tobytes(), s.y.tobytes()) for s in (eng.fetch(q) for q in slots)]
    ref = [(b[0], b[7], b[8]) for b in (_bits([small], ps, True)[0], _bits([large], pl, True)[0])]
    assert got == [ref[0]] * 266 + [ref[1]] * 3
