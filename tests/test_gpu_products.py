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


def _oracle_rows(rp, ri, rx, x):
    from oracle import pdlp_oracle as po
    return po.spmv(rp, ri, rx, x)


def _long_sum_bound(lens, mag):
    """A row of L entries over 256: 256 lanes add L / 256 terms each, then
    trees of depth 5 and 8; every product is rounded once."""
    return (np.ceil(lens / 256.0) + 14) * 2.0 ** -53 * mag


# the row counts around which the rows per warp change (148 * 56 warps times 4,
# 8, 16, 32 rows, and 900,000 rows), with a remainder in the last warp
EDGES = [1, 3, 4, 5, 230, 33_151, 33_153, 66_304, 66_305, 132_607, 265_215, 265_217, 899_999,
         900_000, 900_031]


@pytest.mark.parametrize("m", EDGES)
def test_spmv_rows_per_warp_edges(bk, m):
    """Rows of at most 256 entries equal the oracle's storage-order sum bit for
    bit; longer ones are within the bound of their summation order.  Blocks of
    64 one-entry rows (one run holds them all) and rows of 255, 256 and 257
    entries lie at the start and at the end."""
    rng = np.random.default_rng(m)
    n = 5_000
    lens = rng.integers(0, 5, m)
    special = np.r_[np.ones(128, dtype=np.int64), 255, 256, 257, 0, 300, 90, 90, 90, 1000]
    if m > 2 * special.size:
        lens[:special.size] = special
        lens[-special.size:] = special[::-1]
    rp, ri, rx = _csr(rng, lens, n)
    x = rng.standard_normal(n)
    out = bk.to_device(np.full(m, np.nan))
    for _ in range(2):
        bk.spmv(bk.pointer(rp), bk.index(ri), bk.to_device(rx), bk.to_device(x), out, m)
    got, exp = bk.to_host(out), _oracle_rows(rp, ri, rx, x)
    short = lens <= 256
    assert np.array_equal(got[short], exp[short])
    if not short.all():
        mag = _oracle_rows(rp, ri, np.abs(rx), np.abs(x))
        # the oracle's own sequential sum is off by up to L + 1 roundings
        bound = _long_sum_bound(lens, mag) + (lens + 1) * 2.0 ** -53 * mag
        assert np.all(np.abs(got - exp)[~short] <= bound[~short])


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_chained_products_keep_stream_order(bk, dtype):
    """Each launch starts while the one before it drains: w = A u, u = A^T w, with
    an element-wise kernel between some of them, unsynchronised, equals the
    same chain synchronised after every call, bit for bit."""
    rng = np.random.default_rng(11)
    m, n = 40_000, 70_000
    lens = rng.integers(0, 9, m)
    lens[::5_000] = 700
    rp, ri, rx = _csr(rng, lens, n)
    cols = rng.integers(0, m, 300_000).astype(np.int32)
    cp = np.linspace(0, cols.size, n + 1).astype(np.int64)
    cx = rng.standard_normal(cols.size)
    a = (bk.pointer(rp), bk.index(ri), bk.to_device(rx).to(bk.to_device(np.zeros(1, dtype), dtype).dtype))
    t = (bk.pointer(cp), bk.index(cols), bk.to_device(cx).to(a[2].dtype))
    u0 = bk.to_device(rng.standard_normal(n)).to(a[2].dtype)

    def chain(sync):
        u, w = u0.clone(), bk.empty(m, a[2].dtype)
        for k in range(8):
            bk.spmv(*a, u, w, m)
            if sync:
                bk.sync()
            if k % 2:
                w.mul_(0.25)
            bk.spmv(*t, w, u, n)
            if sync:
                bk.sync()
            u.mul_(0.1)
        bk.sync()
        return bk.to_host(u), bk.to_host(w)

    ref = chain(True)
    for _ in range(3):
        got = chain(False)
        assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])


@pytest.mark.parametrize("m,k", [(2_501, 120), (2_501, 122), (1, 2), (40_000, 6), (40_000, 8)])
def test_spmm_gathers_in_flight(bk, m, k):
    """Both sides of the line (148 * 1024 pairs of columns) between eight and two
    gathers in flight, rows of 0 to 20 entries: the same bits as the flat form,
    which unaligned blocks take."""
    import torch
    rng = np.random.default_rng([m, k])
    n = 300
    rp, ri, rx = _csr(rng, rng.integers(0, 21, m), n)
    args = (bk.pointer(rp), bk.index(ri), bk.to_device(rx))
    X = bk.to_device(rng.standard_normal((n, k)))
    a = bk.empty((m, k))
    bk.spmm(*args, X, a, m, k)
    Xs, Ys = bk.empty(n * k + 1)[1:], bk.empty(m * k + 1)[1:]
    Xs.copy_(X.reshape(-1))
    bk.spmm(*args, Xs, Ys, m, k)
    assert torch.equal(a.reshape(-1), Ys)
