"""The reference's power-iteration start from one kept draw."""

import threading

import numpy as np
import pytest

from sovereign_moe_b200 import pdlp


@pytest.mark.parametrize("n", [0, 1, 2, 3, 64, 65, 2025, 70_000, (1 << 20) - 1, 1 << 20, (1 << 20) + 1])
def test_prefixes_equal_fresh_draws(n):
    for _ in range(2):
        got = pdlp.reference_start(n)
        assert got.shape == (n,) and got.flags.c_contiguous
        assert np.array_equal(got, np.random.default_rng(0).standard_normal(n))


def test_kept_draw_is_read_only_and_bounded():
    pdlp.reference_start(1000)
    pdlp.reference_start((1 << 20) + 5)
    assert pdlp._start.shape[0] <= 1 << 20
    with pytest.raises(ValueError):
        pdlp.reference_start(10)[0] = 1.0


def test_threads():
    want = np.random.default_rng(0).standard_normal(50_000)
    bad = []

    def work(k):
        for n in range(1 + k, 50_000, 4_999):
            if not np.array_equal(pdlp.reference_start(n), want[:n]):
                bad.append((k, n))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
