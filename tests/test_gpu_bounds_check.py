"""The bounds-checked build (``python -m sovereign_moe_b200.build --bounds-check``)
turns a bad index or pointer into ``PDLP_ERR_BOUNDS``, on chip as in the team
engine.

Admission refuses malformed LPs, so the checked build exports a function that
overwrites one entry of an admitted LP, with values that stay inside the slot's
memory.  Skipped with a product build, which has neither."""

import ctypes
import os

import numpy as np
import pytest

from sovereign_moe_b200 import _lib, workloads
from sovereign_moe_b200.batch import BatchEngine
from sovereign_moe_b200.pdlp import PDLPParams

pytestmark = pytest.mark.gpu

DEFINES = _lib.LIB_PATH + ".defines"          # what the library was built with
if not (os.path.exists(DEFINES) and "PDLP_BOUNDS_CHECK" in open(DEFINES).read()):
    pytest.skip("not a bounds-checked build", allow_module_level=True)

LATE = 2          # the test hook that keeps every LP on block teams


def _lp(m, n, per_col):
    rng = np.random.default_rng([m, n])
    cp, ci = workloads.random_structure(rng, m, np.full(n, per_col))
    return workloads.known_optimum(rng, m, n, cp, ci, rng.standard_normal(ci.shape[0])).problem


@pytest.mark.parametrize("hook", [0, LATE])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("which", ["row index", "column index", "row pointer", "column pointer"])
@pytest.mark.parametrize("shape", [(63, 65, 5), (900, 4500, 9)])
def test_a_bad_entry_ends_the_step_with_an_error(shape, which, precision, hook):
    m, n, _ = shape
    prob = _lp(*shape)
    nnz = int(prob.A.nnz)
    kind, at, value = {"row index": (0, nnz - 1, n), "column index": (1, nnz // 2, m),
                       "row pointer": (2, m // 2, nnz), "column pointer": (3, n - 1, 0)}[which]
    params = PDLPParams(device="gpu", eps_abs=0.0, eps_rel=0.0, max_iter=5000, precision=precision)
    with BatchEngine(max_slots=2, test_withhold_arrival=hook) as eng:
        slot = eng.admit(prob, params)
        assert eng.step(50) == 1                    # past the set-up
        _lib.check(eng.lib.pdlp_batch_test_overwrite(eng.h, slot, kind, ctypes.c_int64(at), value))
        with pytest.raises(_lib.PDLPError) as exc:
            eng.step(10)
        assert exc.value.code == _lib.PDLP_ERR_BOUNDS
        with pytest.raises(_lib.PDLPError) as exc:
            eng.step(10)
        assert exc.value.code == _lib.PDLP_ERR_STATE
    with BatchEngine(max_slots=1) as eng:           # the context stays usable
        assert eng.solve_all([prob], PDLPParams(device="gpu", max_iter=64))[0].iterations == 64
