"""Admission of device-resident LPs draws the reference's start vector once for
all of them, also beyond the length that is kept between calls."""

import types

import numpy as np
import pytest

from sovereign_moe_b200 import pdlp
from sovereign_moe_b200.batch import BatchEngine
from sovereign_moe_b200.pdlp import PDLPParams

pytestmark = pytest.mark.gpu


def _device_lp(n, seed):
    """Column j has one entry, in row j mod 2,000; everything a CUDA tensor."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    m, cuda = 2000, "cuda"
    row = torch.arange(n, device=cuda) % m
    order = torch.argsort(row, stable=True)
    cx = torch.rand(n, generator=g, device=cuda, dtype=torch.float64) + 0.1
    rp = torch.zeros(m + 1, dtype=torch.int64, device=cuda)
    torch.cumsum(torch.bincount(row, minlength=m), 0, out=rp[1:])
    A = types.SimpleNamespace(m=m, n=n, nnz=n, cp=torch.arange(n + 1, device=cuda), ci=row.int(),
                              cx=cx, rp=rp, ri=order.int(), rx=cx[order].contiguous())
    zero = torch.zeros(n, dtype=torch.float64, device=cuda)
    b = torch.full((m,), n / m / 8.0, dtype=torch.float64, device=cuda)
    return types.SimpleNamespace(
        A=A, c=torch.randn(n, generator=g, device=cuda, dtype=torch.float64), col_lb=zero,
        col_ub=zero + 1.0, row_lb=b, row_ub=b.clone(), kind=None, obj_offset=0.0, sense=1, Q=None)


def test_one_draw_for_all_lps(require_gpu, monkeypatch):
    n = pdlp._START_KEPT + 100
    probs = [_device_lp(n - 7 * i, i) for i in range(3)] + [_device_lp(1000, 9)]
    params = PDLPParams(device="gpu", max_iter=64)
    with BatchEngine(max_slots=len(probs)) as eng:
        for p in probs:
            eng.admit(p, params)
        eng.run()
        ref = [(s.iterations, s.x.tobytes()) for s in (eng.fetch(i) for i in range(len(probs)))]
    draws = []
    real = np.random.default_rng
    monkeypatch.setattr(np.random, "default_rng", lambda *a: draws.append(a) or real(*a))
    with BatchEngine(max_slots=len(probs)) as eng:
        slots, codes = eng.admit_many(probs, params)
        assert codes == [0] * len(probs) and slots == list(range(len(probs)))
        assert len(draws) == 1
        eng.run()
        assert [(s.iterations, s.x.tobytes()) for s in (eng.fetch(i) for i in slots)] == ref
