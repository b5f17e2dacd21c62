"""The column M2L kernel (mode 5) against the warp-per-target kernel: local
expansions at the orders where its tiles change shape (one and two row tiles,
1 to 4 rows or 8 and 16 per warp tile, the column counts of its shared-memory
plans; level 2 takes one column per lane, level 3 the plan of its order), on
dense levels, target lists and sparse storage."""
from __future__ import annotations

import os
import subprocess
import sys

import numpy as np
import pytest

from wbfmm_b200 import engine, workloads as W

pytestmark = pytest.mark.gpu

LAP, HELM = engine.LAPLACE, engine.HELMHOLTZ


def _problem(problem, order, depth, n, sphere, k):
    p = W.serve_request(np.random.default_rng(order), n, problem == HELM, k, sphere)
    p.depth = depth
    p.order_s = [0] + [order] * depth
    p.order_r = list(p.order_s)
    return p


def _locals(p, precision, mode, **kw):
    cfg = engine.SolverConfig.from_problem(p, precision, **kw)
    with engine.Solver(cfg) as s:
        s.set_m2l_kernel(mode)
        s.set_sources(p.xs).set_strengths(p.q).set_targets(p.xt).run()
        assert all(s.m2l_form(lv) == mode for lv in range(2, p.depth + 1))
        return [s.coefficients(lv)[1] for lv in range(2, p.depth + 1)], s.field()


# tolerances: the two kernels sum the same products in other orders, and a
# level adds up to 189 translations of about 3 (p + 1) products per value: in
# FP64 under 1e-13 of the level's norm, in FP32 a few 1e-6
@pytest.mark.parametrize("precision,tol", [(engine.FP64, 1e-12), (engine.FP32, 2e-5)])
@pytest.mark.parametrize("problem", [LAP, HELM])
@pytest.mark.parametrize("order", [2, 3, 4, 7, 8, 10, 11, 12, 14, 15, 16])
def test_orders(problem, precision, tol, order):
    p = _problem(problem, order, 3, 3001, False, 18.0)
    want, _ = _locals(p, precision, 0)
    got, _ = _locals(p, precision, 5)
    for a, b in zip(got, want):
        assert np.linalg.norm(a - b) < tol * np.linalg.norm(b)


@pytest.mark.parametrize("problem,precision,order", [
    (HELM, engine.FP64, 17), (LAP, engine.FP64, 17), (LAP, engine.FP64, 18), (LAP, engine.FP32, 17),
    (LAP, engine.FP32, 20), (LAP, engine.FP32, 21), (LAP, engine.FP32, 24), (HELM, engine.FP32, 17),
    (HELM, engine.FP32, 18), (HELM, engine.FP32, 19), (HELM, engine.FP32, 20), (HELM, engine.FP32, 24)])
def test_high_orders(problem, precision, order):
    # (k: the FP32 tables of order 24 within their range at level 3)
    p = _problem(problem, order, 3, 3001, False, 40.0)
    want, _ = _locals(p, precision, 0)
    got, _ = _locals(p, precision, 5)
    tol = 1e-12 if precision == engine.FP64 else 2e-5
    for a, b in zip(got, want):
        assert np.linalg.norm(a - b) < tol * np.linalg.norm(b)


@pytest.mark.parametrize("precision,tol", [(engine.FP64, 1e-12), (engine.FP32, 2e-5)])
@pytest.mark.parametrize("problem", [LAP, HELM])
@pytest.mark.parametrize("order", [7, 9, 14])
def test_target_lists_and_sparse(problem, precision, tol, order):
    p = _problem(problem, order, 4, 5003, True, 30.0)
    _, (pot, grad) = _locals(p, precision, 0)
    for kw in (dict(skip_empty=True), dict(sparse=True)):
        _, (f, g) = _locals(p, precision, 5, **kw)
        assert np.linalg.norm(f - pot) < tol * np.linalg.norm(pot)
        assert np.linalg.norm(g - grad) < tol * np.linalg.norm(grad)


@pytest.mark.parametrize("problem,precision,order,forms", [
    (LAP, engine.FP32, 12, [4, 4]), (LAP, engine.FP32, 16, [5, 5]), (LAP, engine.FP64, 12, [3, 5]),
    (HELM, engine.FP32, 4, [2, 2])])
def test_mode_4_is_automatic_elsewhere(problem, precision, order, forms):
    p = _problem(problem, order, 3, 1009, False, 25.0)
    with engine.Solver(engine.SolverConfig.from_problem(p, precision)) as s:
        s.set_m2l_kernel(4)
        s.set_sources(p.xs).set_strengths(p.q).set_targets(p.xt).run()
        assert [s.m2l_form(2), s.m2l_form(3)] == forms


FIRST_USE = r"""
import threading
import numpy as np
from wbfmm_b200 import engine, workloads as W

def solve(problem, order, out, i, start=None):
    p = W.serve_request(np.random.default_rng(order), 2003, problem == engine.HELMHOLTZ, 18.0, False)
    p.depth, p.order_s = 3, [0] + [order] * 3
    p.order_r = list(p.order_s)
    with engine.Solver(engine.SolverConfig.from_problem(p, engine.FP64)) as s:
        s.set_sources(p.xs).set_strengths(p.q).set_targets(p.xt)
        s.build_operators()
        s.synchronize()
        if start is not None:
            start.wait()
        out[i] = s.run().field()

# lanes, columns, and (FP64 Laplace, level 2) tiles
cases = [(engine.LAPLACE, 7), (engine.HELMHOLTZ, 8), (engine.LAPLACE, 12)] * 3
first, again = [None] * len(cases), [None] * len(cases)
start = threading.Barrier(len(cases))
threads = [threading.Thread(target=solve, args=(*c, first, i, start)) for i, c in enumerate(cases)]
for t in threads:
    t.start()
for t in threads:
    t.join()
for i, c in enumerate(cases):
    solve(*c, again, i)
for a, b in zip(first, again):
    assert all(np.array_equal(x, y) for x, y in zip(a, b))
print("same")
"""


def test_first_use_by_several_threads(gpu_lib):
    """The first M2L launches of a process, from several threads on streams of
    their own: each waits for its kernel's table of offsets."""
    r = subprocess.run([sys.executable, "-c", FIRST_USE], capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]
