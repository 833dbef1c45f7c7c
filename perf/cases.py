"""The work that is timed when this engine's speed is judged.

Each case is one call, or one short run of calls, that a user's program makes
through the public entry points: the kernel-level ``Backend``, the planned
sparse product, the batched node relaxation, ``solve_pdlp`` and
``BatchEngine``.  Shapes are those of ``sovereign_moe_b200/workloads.py``:

* ``small``  -- rows at random, every column with ``deg_lo..deg_hi`` entries,
  N(0, 1) values (the 230 x 2,025 single LP, the uneven batch, the served
  stream, the node relaxation);
* ``plan``   -- the multi-period blending plan: banded periods, links to the
  next period, 30 dense coupling rows, values log-uniform in +-[1e-3, 1e3];
* ``power``  -- power-law column degrees (Zipf 1.5, at most 2,000), 1% of the
  rows scaled by 1e4.

Inputs are made on the GPU from the seed, column entries drawn in disjoint row
ranges so that no row repeats.  ``listed()`` has fixed sizes, ``draw(rng)``
others from the same ranges.
"""

import ctypes
import math
from types import SimpleNamespace

import numpy as np
import torch

from sovereign_moe_b200 import PDLPParams, Problem, SparseMatrix, solve_pdlp
from sovereign_moe_b200 import _lib
from sovereign_moe_b200.backend import Backend
from sovereign_moe_b200.batch import BatchEngine
from sovereign_moe_b200.bnr import BNRConfig, BNREngine

PERIODS = 720            # blending plan: periods at 200,000 rows
COUPLING = 30


def listed():
    return [
        # One plain product on a large multi-period plan, as a first-order
        # method written against the kernel-level API makes it.
        dict(name="spmv_plan_f64", path="spmv", shape="plan", m=200_000, n=600_000,
             deg_lo=5, deg_hi=5, side="rows", dtype="f64"),
        # The transposed product of a large power-law LP in float32: the
        # longest pattern, with rows from 1 to 2,000 entries.
        dict(name="spmv_power_t_f32", path="spmv", shape="power", m=1_000_000, n=3_000_000,
             deg_lo=3, deg_hi=4, side="cols", dtype="f32"),
        # A x, then A^T of the result, through plans made once per pattern: the
        # two products of every iteration of a method that keeps its matrix.
        dict(name="planned_pair_f64", path="planned", shape="plan", m=200_000, n=600_000,
             deg_lo=5, deg_hi=5, dtype="f64"),
        # One sparse product against a block of 64 vectors (scenarios, nodes).
        dict(name="spmm_k64", path="spmm", shape="small", m=20_000, n=30_000,
             deg_lo=8, deg_hi=8, k=64),
        # One primal-dual iteration with its step-size sums through the
        # kernel-level API, on a small LP (launch latency) and a large one.
        dict(name="step_small", path="step", shape="small", m=230, n=2_025, deg_lo=6, deg_hi=6),
        dict(name="step_large", path="step", shape="small", m=50_000, n=300_000, deg_lo=3,
             deg_hi=10),
        # Node relaxation: 128 nodes of a 20,000 x 30,000 LP, bound sets and
        # results on the device; and 8 nodes of a small LP through the
        # host-array API, as a tree search's first levels call it.
        dict(name="bnr_wide", path="bnr", shape="small", m=20_000, n=30_000, deg_lo=8, deg_hi=8,
             k=128, iters=60, memory="device"),
        dict(name="bnr_narrow", path="bnr", shape="small", m=2_000, n=3_000, deg_lo=8, deg_hi=8,
             k=8, iters=60, memory="host"),
        # One LP at a time: the small single LP to tolerance from host arrays,
        # the 200,000-row plan for an iteration budget from device arrays (it
        # never reaches a tolerance), and a served mid-size LP in float32.
        dict(name="solve_small", path="solve", shape="small", m=230, n=2_025, deg_lo=6, deg_hi=6,
             precision="fp64", memory="host", max_iter=8_192),
        dict(name="solve_plan", path="solve", shape="plan", m=200_000, n=600_000, deg_lo=5,
             deg_hi=5, precision="fp64", memory="device", max_iter=256),
        dict(name="solve_mid_fp32", path="solve", shape="small", m=10_000, n=40_000, deg_lo=3,
             deg_hi=10, precision="fp32", memory="host", max_iter=1_024),
        # The headline: a batch of uneven LPs in device memory, solved together.
        dict(name="batch_256", path="batch", shape="small", count=256, m_lo=50, m_hi=5_000,
             deg_lo=4, deg_hi=12, max_iter=16_384),
    ]


def draw(rng):
    def logu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(["spmv", "spmv", "planned", "spmm", "step", "bnr", "solve", "solve",
                       "batch"])
    if path in ("spmv", "planned"):
        shape = rng.choice(["plan", "plan", "power", "small"])
        m = logu(2_000, 600_000)
        c = dict(path=path, shape=shape, m=m, n=rng.randint(2, 4) * m + rng.randint(0, 7),
                 dtype=rng.choice(["f64", "f32"]))
        c.update(dict(deg_lo=3, deg_hi=4) if shape == "power" else
                 dict(deg_lo=5, deg_hi=5) if shape == "plan" else dict(deg_lo=3, deg_hi=10))
        if path == "spmv":
            c["side"] = rng.choice(["rows", "cols"])
        return c
    if path == "spmm":
        m = logu(1_000, 40_000)
        return dict(path=path, shape="small", m=m, n=logu(m, 2 * m), deg_lo=8, deg_hi=8,
                    k=logu(1, 160))
    if path == "step":
        m = logu(100, 100_000)
        return dict(path=path, shape="small", m=m, n=rng.randint(2, 8) * m + rng.randint(0, 5),
                    deg_lo=3, deg_hi=10)
    if path == "bnr":
        m = logu(500, 20_000)
        return dict(path=path, shape="small", m=m, n=logu(m, 2 * m), deg_lo=8, deg_hi=8,
                    k=logu(1, 160), iters=rng.choice([20, 40, 60]),
                    memory=rng.choice(["device", "host"]))
    if path == "solve":
        if rng.random() < 0.3:
            m = logu(10_000, 200_000)
            return dict(path=path, shape="plan", m=m, n=3 * m, deg_lo=5, deg_hi=5,
                        precision=rng.choice(["fp64", "fp32"]), memory="device", max_iter=256)
        m = logu(100, 20_000)
        return dict(path=path, shape="small", m=m, n=rng.randint(2, 8) * m, deg_lo=3, deg_hi=10,
                    precision=rng.choice(["fp64", "fp32"]),
                    memory=rng.choice(["host", "device"]), max_iter=1_024)
    return dict(path="batch", shape="small", count=logu(8, 128), m_lo=50, m_hi=logu(500, 5_000),
                deg_lo=4, deg_hi=12, max_iter=4_096)


# ---- inputs ------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _degrees(case, g, m, n):
    if case["shape"] != "power":
        span = case["deg_hi"] - case["deg_lo"] + 1
        return (case["deg_lo"] + (_rand(g, n) * span).long()).clamp(max=m)
    d = _rand(g, n).clamp(min=1e-12).pow(-2.0).floor().clamp(max=2_000.0)
    d = d * (10.0 / 3.0 * n / d.sum().item())
    base = d.floor()
    return (base.long() + (_rand(g, n) < d - base).long()).clamp(1, min(2_000, m))


def _matrix(case, g, m, n):
    """CSC and CSR of A: (cp, ci, cx, rp, ri, rx), on the device."""
    deg = _degrees(case, g, m, n)
    cp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(deg, 0, out=cp[1:])
    nnz = int(cp[-1].item())
    col = torch.repeat_interleave(torch.arange(n, device="cuda"), deg)
    slot = torch.arange(nnz, device="cuda") - cp[col]
    d = deg[col]
    u = _rand(g, nnz)
    if case["shape"] == "plan":
        periods = max(2, PERIODS * m // 200_000)
        prow = m - COUPLING
        edges = torch.linspace(0, prow, periods + 1, device="cuda", dtype=torch.float64).round().long()
        t = col * periods // n
        base, size = edges[t], edges[t + 1] - edges[t]
        lo = base + slot * size // d
        hi = base + (slot + 1) * size // d
        link = (_rand(g, n) < 0.10)[col] & (slot == d - 1) & (t < periods - 1)
        couple = (_rand(g, n) < 0.05)[col] & (slot == d - 2)
        nxt = (t + 1).clamp(max=periods - 1)
        lo = torch.where(link, edges[nxt], lo)
        hi = torch.where(link, edges[nxt + 1], hi)
        lo = torch.where(couple, torch.full_like(lo, prow), lo)
        hi = torch.where(couple, torch.full_like(hi, m), hi)
        val = torch.exp((2.0 * _rand(g, nnz) - 1.0) * math.log(1e3))
        val = torch.where(_rand(g, nnz) < 0.5, -val, val)
    else:
        lo = slot * m // d
        hi = (slot + 1) * m // d
        val = _randn(g, nnz)
    row = lo + torch.minimum((u * (hi - lo)).long(), hi - lo - 1)
    if case["shape"] == "plan":
        order = torch.argsort(col * m + row)
        row, val = row[order], val[order]
    if case["shape"] == "power":
        heavy = _rand(g, m) < 0.01
        val = torch.where(heavy[row], val * 1e4, val)
    order = torch.argsort(row, stable=True)
    rp = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(row, minlength=m), 0, out=rp[1:])
    return (cp, row.int(), val, rp, col[order].int(), val[order].contiguous())


def _product(rp, ri, rx, x):
    """A x by rows in a fixed order (inputs only)."""
    return torch.segment_reduce(rx * x[ri.long()], "sum", offsets=rp, initial=0.0)


def _lp(case, g, m, n):
    """A known-optimum LP: min c'x, Ax = b, 0 <= x <= u.  Returns (problem with
    device tensors, optimal value)."""
    cp, ci, cx, rp, ri, rx = _matrix(case, g, m, n)
    u = 1.0 + 9.0 * _rand(g, n)
    r = _rand(g, n)
    x = (0.1 + 0.8 * _rand(g, n)) * u
    x = torch.where(r < 0.3, torch.zeros_like(x), torch.where(r < 0.6, u, x))
    mag = 0.1 + 0.9 * _rand(g, n)
    z = torch.where(r < 0.3, mag, torch.where(r < 0.6, -mag, torch.zeros_like(mag)))
    b = _product(rp, ri, rx, x)
    c = _product(cp, ci, cx, _randn(g, m)) + z
    prob = SimpleNamespace(
        A=SimpleNamespace(m=m, n=n, nnz=int(ci.numel()), cp=cp, ci=ci, cx=cx, rp=rp, ri=ri, rx=rx),
        c=c, row_lb=b, row_ub=b.clone(), col_lb=torch.zeros_like(u), col_ub=u, kind=None,
        obj_offset=0.0, sense=1, Q=None)
    return prob, float(c.cpu().numpy() @ x.cpu().numpy())


def _host_problem(p):
    h = lambda t: t.cpu().numpy()  # noqa: E731
    A = SparseMatrix(p.A.m, p.A.n, h(p.A.cp), h(p.A.ci), h(p.A.cx), h(p.A.rp), h(p.A.ri), h(p.A.rx))
    return Problem(A=A, c=h(p.c), row_lb=h(p.row_lb), row_ub=h(p.row_ub), col_lb=h(p.col_lb),
                   col_ub=h(p.col_ub), name="case")


def _batch_shapes(case):
    """(rows, columns) of every LP of a batch: the case's, whatever the seed."""
    rng = np.random.default_rng([case["count"], case["m_hi"], 17])
    out = []
    for _ in range(case["count"]):
        m = int(round(math.exp(rng.uniform(math.log(case["m_lo"]), math.log(case["m_hi"])))))
        out.append((m, int(rng.integers(2, 9)) * m))
    return out


def _node_bounds(g, n, k):
    """Bound sets of k branch-and-bound nodes: each halves the box of 3 columns."""
    lo = torch.zeros(n, k, dtype=torch.float64, device="cuda")
    hi = torch.full((n, k), 10.0, dtype=torch.float64, device="cuda")
    j = (_rand(g, 3, k) * n).long()
    up = _rand(g, 3, k) < 0.5
    node = torch.arange(k, device="cuda").expand(3, k)
    hi[j[up], node[up]] = 5.0
    lo[j[~up], node[~up]] = 5.0
    return lo, hi


def _node_problem(case, g):
    m, n = case["m"], case["n"]
    cp, ci, cx, rp, ri, rx = _matrix(case, g, m, n)
    b = _product(rp, ri, rx, _rand(g, n))
    zero = torch.zeros(n, dtype=torch.float64, device="cuda")
    return SimpleNamespace(
        A=SimpleNamespace(m=m, n=n, nnz=int(ci.numel()), cp=cp, ci=ci, cx=cx, rp=rp, ri=ri, rx=rx),
        c=_randn(g, n), row_lb=b, row_ub=b.clone(), col_lb=zero, col_ub=zero + 10.0)


def _step_vectors(case, g):
    m, n = case["m"], case["n"]
    lo = torch.zeros(n, dtype=torch.float64, device="cuda")
    hi = 1.0 + 9.0 * _rand(g, n)
    b = _randn(g, m)
    return dict(x=_rand(g, n) * hi, c=_randn(g, n), aty=_randn(g, n), lo=lo, hi=hi,
                sumx=torch.zeros_like(lo), y=_randn(g, m), ax=_randn(g, m), rl=b - 0.1, ru=b + 0.1,
                sumy=torch.zeros_like(b))


def _params(case):
    return PDLPParams(eps_abs=1e-6, eps_rel=1e-6, device="gpu", max_iter=case["max_iter"],
                      precision=case.get("precision", "fp64"))


# ---- prepare and run ------------------------------------------------------------


def prepare(case, seed):
    g = _generator(seed)
    path = case["path"]
    s = SimpleNamespace(path=path)
    if path in ("spmv", "planned", "spmm", "step"):
        m, n = case["m"], case["n"]
        s.m, s.n, s.bk = m, n, Backend("gpu")
        s.cp, s.ci, s.cx, s.rp, s.ri, s.rx = _matrix(case, g, m, n)
    if path == "spmv":
        dt = torch.float32 if case["dtype"] == "f32" else torch.float64
        if case["side"] == "cols":
            s.m, s.n, s.rp, s.ri, s.rx = n, m, s.cp, s.ci, s.cx
        s.rx = s.rx.to(dt)
        s.x = _randn(g, s.n).to(dt)
        s.out = torch.empty(s.m, dtype=dt, device="cuda")
    elif path == "planned":
        dt = torch.float32 if case["dtype"] == "f32" else torch.float64
        s.rx, s.cx = s.rx.to(dt), s.cx.to(dt)
        s.x = _randn(g, n).to(dt)
        s.y = torch.empty(m, dtype=dt, device="cuda")
        s.z = torch.empty(n, dtype=dt, device="cuda")
        s.rows = s.bk.spmv_plan(s.rp, s.ri, m, n)
        s.cols = s.bk.spmv_plan(s.cp, s.ci, n, m)
    elif path == "spmm":
        s.k = case["k"]
        s.X = _randn(g, n, s.k)
        s.Y = torch.empty(m, s.k, dtype=torch.float64, device="cuda")
    elif path == "step":
        for name, v in _step_vectors(case, g).items():
            setattr(s, name, v)
        new = lambda k: torch.empty(k, dtype=torch.float64, device="cuda")  # noqa: E731
        s.dx, s.ady, s.dy, s.adx = new(n), new(n), new(m), new(m)
    elif path == "bnr":
        p = _node_problem(case, g)
        s.iters, s.k, s.device = case["iters"], case["k"], case["memory"] == "device"
        s.eng = BNREngine(_host_problem(p), None, BNRConfig(batch=s.k, iters=s.iters, device="gpu"))
        s.lo, s.hi = _node_bounds(g, case["n"], s.k)
        if s.device:
            new = lambda *d: torch.empty(*d, dtype=torch.float64, device="cuda")  # noqa: E731
            s.bounds, s.x, s.y = new(s.k), new(case["n"], s.k), new(case["m"], s.k)
        else:
            s.lo, s.hi = s.lo.cpu().numpy(), s.hi.cpu().numpy()
    elif path == "solve":
        p, _ = _lp(case, g, case["m"], case["n"])
        s.prob = p if case["memory"] == "device" else _host_problem(p)
        s.params = _params(case)
    else:
        s.probs = [_lp(case, g, m, n)[0] for m, n in _batch_shapes(case)]
        s.params = _params(case)
        s.eng = BatchEngine(max_slots=case["count"])
    return s


def run(s):
    if s.path == "spmv":
        return s.bk.spmv(s.rp, s.ri, s.rx, s.x, s.out, s.m)
    if s.path == "planned":
        s.bk.spmv_planned(s.rows, s.rx, s.x, s.y)
        s.bk.spmv_planned(s.cols, s.cx, s.y, s.z)
        return s.y, s.z
    if s.path == "spmm":
        return s.bk.spmm(s.rp, s.ri, s.rx, s.X, s.Y, s.m, s.k)
    if s.path == "step":
        return _step(s)
    if s.path == "bnr":
        return _bnr(s)
    if s.path == "solve":
        sol = solve_pdlp(s.prob, s.params)
        return dict(x=sol.x, y=sol.y, d=sol.reduced_costs, objective=np.array([sol.info.primal_obj]),
                    iterations=int(sol.iterations), status=int(sol.status))
    sols = s.eng.solve_all(s.probs, s.params)
    return dict(x=np.concatenate([v.x for v in sols]), y=np.concatenate([v.y for v in sols]),
                d=np.concatenate([v.reduced_costs for v in sols]),
                objective=np.array([v.info.primal_obj for v in sols]),
                iterations=np.array([v.iterations for v in sols]),
                status=np.array([int(v.status) for v in sols]))


TAU, SIGMA, ETA = 0.05, 0.05, 0.05


def _step(s):
    """One fused primal-dual iteration and the sums of the step-size test."""
    bk = s.bk
    bk.pdhg_primal(s.x, s.dx, s.c, s.aty, s.lo, s.hi, TAU, s.n)
    bk.spmv(s.rp, s.ri, s.rx, s.dx, s.adx, s.m)
    bk.pdhg_dual(s.y, s.dy, s.ax, s.adx, s.rl, s.ru, SIGMA, s.m)
    bk.spmv(s.cp, s.ci, s.cx, s.dy, s.ady, s.n)
    bk.pdhg_accum(s.aty, s.ady, s.sumx, s.x, ETA, s.n)
    sums = np.array([bk.dot(s.dy, s.adx), bk.nrm2(s.dx), bk.nrm2(s.dy), bk.nrm_inf(s.dx)])
    return dict(x=s.x, y=s.y, ax=s.ax, aty=s.aty, dx=s.dx, dy=s.dy, sumx=s.sumx, sums=sums)


def _bnr(s):
    if not s.device:
        r = s.eng.solve_batch(s.lo, s.hi)
        return r.bounds, r.x, r.y
    cfg = s.eng.cfg
    _lib.check(s.eng.lib.pdlp_bnr_solve_batch(
        s.eng.h, s.k, s.lo.data_ptr(), s.hi.data_ptr(), None, None, s.iters,
        ctypes.c_double(cfg.step_growth), ctypes.c_double(cfg.step_damp), s.bounds.data_ptr(),
        s.x.data_ptr(), s.y.data_ptr(), None, _lib.PDLP_MEM_DEVICE))
    return s.bounds, s.x, s.y


# ---- work and exact values ---------------------------------------------------


def _nnz(case, n):
    if case["shape"] == "power":
        return 10.0 / 3.0 * n
    return 0.5 * (case["deg_lo"] + case["deg_hi"]) * n


def work(case):
    path = case["path"]
    if path == "batch":
        rows = (case["m_hi"] - case["m_lo"]) / math.log(case["m_hi"] / case["m_lo"])
        m, n = case["count"] * rows, case["count"] * 5.0 * rows
    else:
        m, n = case["m"], case["n"]
    nnz = _nnz(case, n)
    if path in ("spmv", "planned"):
        w = 4 if case["dtype"] == "f32" else 8
        one = (w + 4) * nnz + w * (m + n)
        if path == "planned":
            return dict(bytes=2 * one + 8 * (m + n), flops=4.0 * nnz)
        return dict(bytes=one + 8 * (m if case["side"] == "rows" else n), flops=2.0 * nnz)
    if path == "spmm":
        return dict(bytes=12 * nnz + 8 * m + 8.0 * case["k"] * (m + n), flops=2.0 * nnz * case["k"])
    if path == "step":
        # both copies of the matrix; x, c, aty, lo, hi, sum_x and y, ax, rl, ru
        # in; x, dx, aty, sum_x and y, dy, ax out
        return dict(bytes=24 * nnz + 8 * (m + n) + 8 * (10.0 * n + 7.0 * m), flops=4.0 * nnz)
    if path == "bnr":
        k = case["k"]
        return dict(bytes=24 * nnz + 8.0 * k * (3 * n + m),
                    flops=case["iters"] * k * (4.0 * nnz + 12.0 * (m + n)))
    # the LP read once and its solution written once; the products of the
    # iterations, at the budget or at about the median count of a batch
    iters = 1_500 if path == "batch" else min(case["max_iter"], 600)
    return dict(bytes=24 * nnz + 8 * (m + n) + 8 * (3.0 * m + 5.0 * n), flops=4.0 * iters * nnz)


def exact(case, seed):
    path = case["path"]
    g = _generator(seed)
    if path == "batch":
        best = [_lp(case, g, m, n)[1] for m, n in _batch_shapes(case)]
        # an LP that stops at the iteration budget has no objective to report
        return dict(x=None, y=None, d=None, objective=None if case["max_iter"] < 16_384
                    else np.array(best), iterations=None, status=None)
    if path == "solve":
        if case["max_iter"] < 8_192:
            return None
        best = _lp(case, g, case["m"], case["n"])[1]
        return dict(x=None, y=None, d=None, objective=np.array([best]), iterations=None,
                    status=None)
    if path == "bnr":
        return None
    m, n = case["m"], case["n"]
    cp, ci, cx, rp, ri, rx = _matrix(case, g, m, n)
    if path == "spmv":
        dt = torch.float32 if case["dtype"] == "f32" else torch.float64
        if case["side"] == "cols":
            m, n, rp, ri, rx = n, m, cp, ci, cx
        return _rows(m, rp, ri, rx.to(dt), _randn(g, n).to(dt))
    if path == "planned":
        dt = torch.float32 if case["dtype"] == "f32" else torch.float64
        y = _rows(m, rp, ri, rx.to(dt), _randn(g, n).to(dt))
        return y, _rows(n, cp, ci, cx.to(dt), y)
    if path == "spmm":
        X = _randn(g, n, case["k"]).cpu()
        row = torch.repeat_interleave(torch.arange(m), torch.diff(rp).cpu())
        out = torch.zeros(m, case["k"], dtype=torch.float64)
        for k in range(0, case["k"], 16):
            out[:, k:k + 16].index_add_(0, row, rx.cpu()[:, None] * X[ri.cpu().long(), k:k + 16])
        return out
    v = {k: t.cpu().numpy() for k, t in _step_vectors(case, g).items()}
    xn = np.clip(v["x"] - TAU * (v["c"] + v["aty"]), v["lo"], v["hi"])
    dx = xn - v["x"]
    adx = _rows(m, rp, ri, rx, dx).numpy()
    ax = v["ax"] + adx
    w = v["y"] + SIGMA * (ax + adx)
    yn = w - SIGMA * np.clip(w / SIGMA, v["rl"], v["ru"])
    dy = yn - v["y"]
    aty = v["aty"] + _rows(n, cp, ci, cx, dy).numpy()
    sums = np.array([dy @ adx, np.linalg.norm(dx), np.linalg.norm(dy),
                     np.abs(dx).max(initial=0.0)])
    return dict(x=xn, y=yn, ax=ax, aty=aty, dx=dx, dy=dy, sumx=v["sumx"] + ETA * xn, sums=sums)


def _rows(m, rp, ri, rx, x):
    """A x in 64 bits on the host."""
    h = lambda t: t.double().cpu().numpy() if torch.is_tensor(t) else np.asarray(t, np.float64)  # noqa: E731
    row = np.repeat(np.arange(m), np.diff(rp.cpu().numpy()))
    return torch.from_numpy(np.bincount(row, weights=h(rx) * h(x)[ri.cpu().numpy()], minlength=m))
