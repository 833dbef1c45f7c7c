"""The one-launch reductions (``pdlp_dot``, ``pdlp_nrm2``, ``pdlp_nrm_inf``)
at the sizes where their grid, their unrolled loop and their last block change,
and with more calls in flight than the scratch slots the library keeps.

A sum of n terms added by 592 x 256 threads and then by trees of depth at most
32 is off by at most (ceil(n / (592 * 256)) + 32) rounding errors of the sum of
magnitudes; ``math.fsum`` gives the exact sum of the rounded products, which
adds one more."""

import math
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STRIDE = 592 * 256
SIZES = [1, 31, 32, 255, 256, 257, 2025, STRIDE - 1, STRIDE, STRIDE + 1, 4 * STRIDE - 1,
         4 * STRIDE, 4 * STRIDE + 257, 9 * STRIDE + 3]


@pytest.fixture(scope="module")
def bk():
    from sovereign_moe_b200.backend import Backend
    return Backend("gpu")


def _bound(n, mag):
    return (math.ceil(n / STRIDE) + 33) * 2.0 ** -53 * mag


@pytest.mark.parametrize("n", SIZES)
def test_reductions_at_the_edges_of_the_grid(bk, n):
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal(n), rng.standard_normal(n)
    ag, bg = bk.to_device(a), bk.to_device(b)
    assert abs(bk.dot(ag, bg) - math.fsum(a * b)) <= _bound(n, math.fsum(np.abs(a * b)))
    sq = math.fsum(a * a)
    assert abs(bk.nrm2(ag) ** 2 - sq) <= _bound(n, sq) + 4 * 2.0 ** -53 * sq   # root and square
    assert bk.nrm_inf(ag) == np.abs(a).max()
    assert bk.dot(ag, bg) == bk.dot(ag, bg)


def test_reductions_of_one_negative_or_nonfinite_element(bk):
    for v in (-3.0, 0.0, -0.0):
        assert bk.nrm_inf(bk.to_device(np.array([v]))) == abs(v)
        assert bk.nrm2(bk.to_device(np.array([v]))) == abs(v)
    assert bk.nrm_inf(bk.to_device(np.array([1.0, -np.inf]))) == np.inf
    assert math.isnan(bk.dot(bk.to_device(np.array([np.nan, 1.0])),
                             bk.to_device(np.array([1.0, 1.0]))))


def test_reductions_from_many_threads_and_streams(bk):
    """24 threads on streams of their own, 20 calls each, with at most 16
    scratch slots kept: every result is the thread's own."""
    import torch
    n = 70_001
    vecs = [bk.to_device(np.full(n, float(t + 1))) for t in range(24)]
    ones = bk.to_device(np.ones(n))
    torch.cuda.synchronize()
    wrong = []

    def work(t):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                got = (bk.dot(vecs[t], ones), bk.nrm_inf(vecs[t]))
                if got != (n * float(t + 1), float(t + 1)):
                    wrong.append((t, got))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(24)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not wrong
