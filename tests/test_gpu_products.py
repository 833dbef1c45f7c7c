"""Sparse products at the sizes where their launch shapes change.

The dense-block product (``pdlp_spmm_f64``) sums each entry of a row in storage
order with fused multiply-adds, whatever its block shape, so its error against
the exact sum is at most one rounding per entry."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bk():
    from sovereign_moe_b200.backend import Backend
    return Backend("gpu")


def _csr(rng, lens, n):
    rp = np.zeros(len(lens) + 1, dtype=np.int64)
    np.cumsum(lens, out=rp[1:])
    return rp, rng.integers(0, n, rp[-1]).astype(np.int32), rng.standard_normal(rp[-1])


@pytest.mark.parametrize("k", [1, 2, 3, 4, 31, 32, 33, 62, 63, 64, 65, 66, 127, 128, 130, 257])
def test_spmm_widths(bk, k):
    rng = np.random.default_rng(k)
    n = 97
    lens = np.r_[0, 1, 2, 3, 4, 5, 7, 8, 9, 63, 200, 0, rng.integers(0, 12, 61)]
    rp, ri, rx = _csr(rng, lens, n)
    m = len(lens)
    X = rng.standard_normal((n, k))
    out = bk.to_device(np.full((m, k), np.nan))
    bk.spmm(bk.pointer(rp), bk.index(ri), bk.to_device(rx), bk.to_device(X), out, m, k)
    got = bk.to_host(out)
    for r in range(m):
        s = slice(rp[r], rp[r + 1])
        terms = rx[s, None].astype(np.longdouble) * X[ri[s]].astype(np.longdouble)
        bound = (int(lens[r]) + 1) * 2.0 ** -53 * np.abs(terms).sum(axis=0)
        assert np.all(np.abs(got[r] - terms.sum(axis=0)) <= bound)


def test_spmm_unaligned_blocks_equal_aligned_ones(bk):
    """X and Y at 8 bytes past a 16-byte boundary take the one-column form,
    which gives the same bits."""
    import torch
    rng = np.random.default_rng(5)
    m, n, k = 40, 30, 34
    rp, ri, rx = _csr(rng, rng.integers(0, 20, m), n)
    args = (bk.pointer(rp), bk.index(ri), bk.to_device(rx))
    X = bk.to_device(rng.standard_normal((n, k)))
    a = bk.empty((m, k))
    bk.spmm(*args, X, a, m, k)
    Xs, Ys = bk.empty(n * k + 1)[1:], bk.empty(m * k + 1)[1:]
    Xs.copy_(X.reshape(-1))
    bk.spmm(*args, Xs, Ys, m, k)
    assert torch.equal(a.reshape(-1), Ys)
