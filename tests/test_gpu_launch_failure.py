"""A launch that fails while clusters of the same step run (made to fail on the
host, by the test hook): the step waits for those clusters and returns the
error, and the batch refuses later calls; the context stays usable."""

import numpy as np
import pytest

from sovereign_moe_b200 import _lib, workloads
from sovereign_moe_b200.batch import BatchEngine
from sovereign_moe_b200.pdlp import PDLPParams

pytestmark = pytest.mark.gpu

LAUNCH_FAILS = 3


def _lp(m, n, per_col):
    rng = np.random.default_rng([m, n])
    cp, ci = workloads.random_structure(rng, m, np.full(n, per_col))
    return workloads.known_optimum(rng, m, n, cp, ci, rng.standard_normal(ci.shape[0])).problem


def _params(**kw):
    return PDLPParams(device="gpu", eps_abs=0.0, eps_rel=0.0, max_iter=3000, **kw)


SMALL, LARGE, BEYOND = (63, 65, 5), (1400, 7000, 8), (2300, 9100, 8)


# two cluster sizes, on streams of their own; the same beside an LP for the team
# engine; one size in two precisions, on the batch's stream
@pytest.mark.parametrize("lps", [[(SMALL, "fp64")] * 20 + [(LARGE, "fp64")],
                                 [(SMALL, "fp64")] * 20 + [(LARGE, "fp64"), (BEYOND, "fp64")],
                                 [(SMALL, "fp64"), (SMALL, "fp32")]])
def test_a_failed_launch_beside_running_clusters(lps):
    probs = [(_lp(*s), p) for s, p in lps]
    with BatchEngine(max_slots=len(probs), test_withhold_arrival=LAUNCH_FAILS) as eng:
        for p, precision in probs:
            eng.admit(p, _params(precision=precision))
        with pytest.raises(_lib.PDLPError) as exc:
            eng.step(1 << 12)
        assert exc.value.code == _lib.PDLP_ERR_CUDA
        for call in (lambda: eng.step(64), lambda: eng.admit(probs[0][0], _params())):
            with pytest.raises(_lib.PDLPError) as exc:
                call()
            assert exc.value.code == _lib.PDLP_ERR_STATE
    with BatchEngine(max_slots=1) as eng:
        assert eng.solve_all([probs[0][0]], PDLPParams(device="gpu", max_iter=64))[0].iterations == 64


def test_the_first_launch_is_not_affected():
    prob = _lp(63, 65, 5)
    with BatchEngine(max_slots=1, test_withhold_arrival=LAUNCH_FAILS) as eng:
        got = eng.solve_all([prob], _params())[0]
    with BatchEngine(max_slots=1) as eng:
        ref = eng.solve_all([prob], _params())[0]
    assert np.array_equal(got.x, ref.x) and np.array_equal(got.y, ref.y)
