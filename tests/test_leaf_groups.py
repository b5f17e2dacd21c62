"""The forms of P2M against each other: a warp per leaf box against 8 lanes
(trees of few points per leaf) and against a CTA (few leaves of many points).
The rule changes sides at 12 and at 48 points per leaf on average, so a problem
on the line and the same problem with one more source, of strength zero, take
two forms."""
from __future__ import annotations

import numpy as np
import pytest

from wbfmm_b200 import engine

pytestmark = pytest.mark.gpu

LAP, HELM = engine.LAPLACE, engine.HELMHOLTZ


def _compare(problem, precision, order, dipoles, depth, n, forms, tol):
    rng = np.random.default_rng(order)
    w = 2 if problem == HELM else 1
    assert forms == tuple(engine.selftest_p2m_lanes(problem, precision, order, 8 ** depth, m)
                          for m in (n, n + 1))
    pts = rng.uniform(-0.5, 0.5, (n, 3))
    pts[:40] = rng.uniform(0.3, 0.31, (40, 3))          # one leaf with more points than lanes
    q, d = rng.standard_normal((n, w)), rng.standard_normal((n, w))
    nrm = rng.standard_normal((n, 3))
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    orders = [0] + [order] * depth
    cfg = engine.SolverConfig(problem, depth, orders, list(orders), 16.0, (-0.51,) * 3, 1.02, precision)

    def leaves(extra):
        z = np.zeros((extra, w))
        p = np.concatenate([pts, np.full((extra, 3), -0.3)])
        m = np.concatenate([nrm, np.tile([0.0, 0.0, 1.0], (extra, 1))])
        with engine.Solver(cfg) as s:
            s.set_sources(p, m if dipoles else None)
            s.set_strengths(np.concatenate([q, z]).ravel(),
                            np.concatenate([d, z]).ravel() if dipoles else None)
            s.set_targets(pts)
            s.leaf_expansions()
            return s.coefficients(depth)[0]

    on, past = leaves(0), leaves(1)
    assert np.linalg.norm(on - past) < tol * np.linalg.norm(past)


# both forms add a leaf's at most few dozen terms of like size in another
# order: a few units of rounding of the level's norm
@pytest.mark.parametrize("precision,tol", [(engine.FP64, 1e-14), (engine.FP32, 2e-6)])
@pytest.mark.parametrize("problem", [LAP, HELM])
@pytest.mark.parametrize("order", [2, 6, 14, 17])
@pytest.mark.parametrize("dipoles", [False, True])
def test_p2m_forms(gpu_lib, problem, precision, tol, order, dipoles):
    if problem == HELM and precision == engine.FP64:    # 8 lanes up to order 13
        order = {14: 12, 17: 13}.get(order, order)
    _compare(problem, precision, order, dipoles, 4, 12 * 4096, (8, 32), tol)


# (the sums of a few hundred terms: ten units)
@pytest.mark.parametrize("precision,tol", [(engine.FP64, 2e-14), (engine.FP32, 4e-6)])
@pytest.mark.parametrize("problem", [LAP, HELM])
@pytest.mark.parametrize("order,dipoles", [(2, False), (6, True), (14, False), (14, True), (24, False)])
@pytest.mark.parametrize("depth,per", [(2, 48), (3, 48)])
def test_p2m_shared(gpu_lib, problem, precision, tol, order, dipoles, depth, per):
    _compare(problem, precision, order, dipoles, depth, per * 8 ** depth, (32, 128), tol)
