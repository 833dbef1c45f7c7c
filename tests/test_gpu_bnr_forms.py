"""The fused and the split form of a node-relaxation iteration.

Both make the reference's operations in the same order and add the per-node sums
in the same fixed tree, so either equals the tree-order oracle bit for bit.
Which form runs depends on the rows and the nodes; the sizes here lie on both
sides of every line of that rule, with odd and even node counts, row blocks
whose entries do not fit the staging buffer, empty rows and columns, and a
ragged last block."""

from types import SimpleNamespace

import numpy as np
import pytest

from oracle.bnr_oracle import BNROracle
from sovereign_moe_b200.bnr import BNRConfig, BNREngine
from sovereign_moe_b200.problem import SparseMatrix

pytestmark = pytest.mark.gpu


def _problem(m, n, per_col, seed, dense_rows=0):
    rng = np.random.default_rng([m, n, seed])
    cols = np.repeat(np.arange(n), per_col)
    rows = rng.integers(0, m, cols.size)
    if dense_rows:
        rows = np.concatenate([rows, np.repeat(np.arange(dense_rows), n)])
        cols = np.concatenate([cols, np.tile(np.arange(n), dense_rows)])
    if n > 3:                                  # an empty column
        keep = cols != n // 2
        rows, cols = rows[keep], cols[keep]
    A = SparseMatrix.from_triplets(rows, cols, rng.standard_normal(rows.size), m, n)
    b = A.matvec(rng.random(n))
    prob = SimpleNamespace(A=A, c=rng.standard_normal(n), row_lb=b, row_ub=b + 0.5, col_lb=None,
                           col_ub=None, obj_offset=0.25)
    return prob, rng


def _check(prob, rng, k, iters):
    m, n = prob.A.m, prob.A.n
    lo = np.where(rng.random((n, k)) < 0.1, 2.0, 0.0)
    hi = np.where(rng.random((n, k)) < 0.1, 4.0, 8.0)
    A = prob.A
    eng = BNREngine(prob, SimpleNamespace(obj=2.0), BNRConfig(batch=k, iters=iters, device="gpu"))
    ora = BNROracle(A.rp, A.ri, A.rx, A.cp, A.ci, A.cx, prob.c, prob.row_lb, prob.row_ub, 2.0, 0.25,
                    batch=k, iters=iters, sum_order="tree")
    for _ in range(2):                         # the second call goes on with the step sizes
        r, o = eng.solve_batch(lo, hi), ora.solve_batch(lo, hi)
        for a, b in ((r.x, o.x), (r.y, o.y), (r.bounds, o.bounds)):
            a, b = np.asarray(a), np.asarray(b)
            assert np.array_equal(a, b, equal_nan=True), float(np.nanmax(np.abs(a - b)))
        assert np.array_equal(eng.step_sizes(k)[0], ora.eta[:k])
    eng.close()


@pytest.mark.parametrize("k", [1, 2, 3, 4, 7, 8, 9, 15, 16, 17, 18, 64, 65])
def test_node_counts(k):
    prob, rng = _problem(70, 131, 5, k)
    _check(prob, rng, k, 12)


@pytest.mark.parametrize("m,n", [(1, 1), (63, 64), (64, 65), (129, 1)])
def test_row_blocks(m, n):
    prob, rng = _problem(m, n, min(3, m), 1)
    _check(prob, rng, 6, 9)


def test_rows_beyond_the_staging_buffer():
    prob, rng = _problem(90, 700, 4, 2, dense_rows=3)
    for k in (5, 12):
        _check(prob, rng, k, 8)


# blocks of 64 rows times tiles of nodes: 219 blocks x 1 tile (four threads), 219 x
# 2 -> eight threads, 219 x 3 (eight), 219 x 4 > 800 -> split; odd: 219 x 3 and split
@pytest.mark.parametrize("k", [8, 16, 48, 64, 3, 24, 33])
def test_both_sides_of_the_line(k):
    prob, rng = _problem(6_000, 8_000, 3, 3)
    _check(prob, rng, k, 4)
