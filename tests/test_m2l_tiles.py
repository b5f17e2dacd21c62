"""The offset-major tile M2L at the orders and levels that the automatic choice
still gives it (above the columns' orders, and level 2 of a dense FP64 Laplace
solve), on dense levels, target lists and sparse storage, and forced (mode 3)
below, against the warp-per-target kernel; its scaled Helmholtz form against
the FP64 solve."""
from __future__ import annotations

import numpy as np
import pytest

from wbfmm_b200 import engine, workloads as W

pytestmark = pytest.mark.gpu

LAP, HELM = engine.LAPLACE, engine.HELMHOLTZ


def _problem(problem, order, depth):
    p = W.serve_request(np.random.default_rng(order), 3001, problem == HELM, 40.0, True)
    p.depth = depth
    p.order_s = [0] + [order] * depth
    p.order_r = list(p.order_s)
    return p


def _solve(p, precision, mode, forms, **kw):
    """Fields, the kernels of levels 2.. checked where forms are given."""
    with engine.Solver(engine.SolverConfig.from_problem(p, precision, **kw)) as s:
        s.set_m2l_kernel(mode)
        s.set_sources(p.xs).set_strengths(p.q).set_targets(p.xt).run()
        assert forms is None or [s.m2l_form(lv) for lv in range(2, p.depth + 1)] == forms
        return s.field()


def _close(got, want, tol):
    for a, b in zip(got, want):
        assert np.linalg.norm(a - b) < tol * np.linalg.norm(b)


# tolerances: as for the columns (test_m2l_cols.py), the same sums in another order
@pytest.mark.parametrize("kw", [{}, dict(skip_empty=True), dict(sparse=True)])
@pytest.mark.parametrize("problem,precision,order", [
    (HELM, engine.FP64, 18), (LAP, engine.FP64, 19), (LAP, engine.FP64, 20),
    (HELM, engine.FP32, 25), (LAP, engine.FP32, 25)])
def test_above_the_columns(problem, precision, order, kw):
    p = _problem(problem, order, 3)
    tol = 1e-12 if precision == engine.FP64 else 2e-5
    _close(_solve(p, precision, 1, [3, 3], **kw), _solve(p, precision, 0, [0, 0]), tol)


@pytest.mark.parametrize("skip", [False, True])
@pytest.mark.parametrize("order", [10, 14, 18])
def test_level_2(order, skip):
    p = _problem(LAP, order, 3)
    _close(_solve(p, engine.FP64, 1, [3, 5], skip_empty=skip), _solve(p, engine.FP64, 0, [0, 0]), 1e-12)


# 3: tiles wherever they fit, also where columns do
@pytest.mark.parametrize("kw", [{}, dict(skip_empty=True), dict(sparse=True)])
@pytest.mark.parametrize("precision", [engine.FP64, engine.FP32])
@pytest.mark.parametrize("problem,order", [(LAP, 3), (LAP, 14), (HELM, 4), (HELM, 14)])
def test_forced(problem, order, precision, kw):
    p = _problem(problem, order, 3)
    tol = 1e-12 if precision == engine.FP64 else 2e-5
    _close(_solve(p, precision, 3, [3, 3], **kw), _solve(p, precision, 0, [0, 0]), tol)


# the scaled form's bound against FP64 is that of the range rule's admission
@pytest.mark.parametrize("kw", [{}, dict(skip_empty=True), dict(sparse=True)])
@pytest.mark.parametrize("mode", [3, 5])
def test_scaled_helmholtz(mode, kw):
    p = W.serve_request(np.random.default_rng(91), 60_000, True, 7.0, True)
    p.depth = 4
    p.order_s = p.order_r = [0] + [14] * 4
    assert 0.8 <= 2 * 7.0 * p.D / 16 < 1.02          # scaled at the leaf level
    _close(_solve(p, engine.FP32, mode, [mode] * 3, **kw), _solve(p, engine.FP64, mode, None), 1.5e-6)
