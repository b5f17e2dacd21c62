"""The forms of P2M against each other: a warp per leaf box against 8 lanes (many
leaves of few points) and against a CTA (few leaves of many points).  Each pair
of problems lies on either side of a line of the rule and differs by one
source, of strength zero."""
from __future__ import annotations

import numpy as np
import pytest

from wbfmm_b200 import engine

pytestmark = pytest.mark.gpu

LAP, HELM = engine.LAPLACE, engine.HELMHOLTZ


def _compare(problem, precision, order, dipoles, depth, pts, extra, forms, tol, **kw):
    """Leaf expansions of pts and of pts and the point extra."""
    rng = np.random.default_rng(order)
    n, w = len(pts), 2 if problem == HELM else 1
    q, d = rng.standard_normal((n, w)), rng.standard_normal((n, w))
    nrm = rng.standard_normal((n, 3))
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    orders = [0] + [order] * depth
    cfg = engine.SolverConfig(problem, depth, orders, list(orders), 16.0, (-0.51,) * 3, 1.02,
                              precision, **kw)

    def leaves(more):
        z = np.zeros((more, w))
        p = np.concatenate([pts, np.tile(extra, (more, 1))])
        m = np.concatenate([nrm, np.tile([0.0, 0.0, 1.0], (more, 1))])
        with engine.Solver(cfg) as s:
            s.set_sources(p, m if dipoles else None)
            s.set_strengths(np.concatenate([q, z]).ravel(),
                            np.concatenate([d, z]).ravel() if dipoles else None)
            s.set_targets(pts)
            s.leaf_expansions()
            assert s.p2m_form() == forms[more]
            return s.coefficients(depth)[0]

    a, b = leaves(0), leaves(1)
    assert np.linalg.norm(a - b) < tol * np.linalg.norm(b)


W5 = 1.02 / 32          # leaf width at depth 5


def _few_points():
    """Four points per leaf of depth 5 on average, 32 in one leaf, and 20 in a
    leaf whose siblings are empty."""
    rng = np.random.default_rng(3)
    pts = rng.uniform(-0.5, 0.5, (4 * 8 ** 5, 3))
    cell = np.floor((pts + 0.51) / W5).astype(int)
    full, lone = np.array([25, 25, 25]), np.array([8, 10, 12])
    pts = pts[~(np.all(cell == full, 1) | np.all(cell // 2 == lone // 2, 1))]
    inside = rng.uniform(0.05, 0.95, (52, 3)) * W5 - 0.51
    return np.concatenate([pts, inside[:32] + full * W5, inside[32:] + lone * W5])


# both forms add a leaf's at most few dozen terms of like size in another
# order: a few units of rounding of the level's norm
@pytest.mark.parametrize("precision,tol", [(engine.FP64, 1e-14), (engine.FP32, 2e-6)])
@pytest.mark.parametrize("problem", [LAP, HELM])
@pytest.mark.parametrize("order", [2, 6, 14, 17])
@pytest.mark.parametrize("dipoles", [False, True])
def test_p2m_forms(gpu_lib, problem, precision, tol, order, dipoles):
    if problem == HELM and precision == engine.FP64:    # 8 lanes up to order 13
        order = {14: 12, 17: 13}.get(order, order)
    _compare(problem, precision, order, dipoles, 5, _few_points(), np.full(3, 25.5 * W5 - 0.51),
             (8, 32), tol)


# leaves of 17 to 32 points need 24 occupied groups of four leaves per SM: one
# leaf of each of 3551 parents, and of one parent more; up to 16 none
@pytest.mark.parametrize("kw", [{}, dict(skip_empty=True)])
@pytest.mark.parametrize("full,forms", [(17, (32, 8)), (16, (8, 8))])
@pytest.mark.parametrize("problem,precision,tol", [(LAP, engine.FP32, 2e-6), (HELM, engine.FP64, 1e-14)])
def test_p2m_occupied_groups(gpu_lib, problem, precision, tol, full, forms, kw):
    rng = np.random.default_rng(4)
    ijk = np.stack(np.meshgrid(*[np.arange(16)] * 3, indexing="ij"), -1).reshape(-1, 3)
    ijk = rng.permutation(ijk)
    pts = (2 * ijk + 0.4) * W5 - 0.51
    more = (2 * ijk[0] + rng.uniform(0.1, 0.9, (full - 1, 3))) * W5 - 0.51
    _compare(problem, precision, 6, False, 5, np.concatenate([pts[:3551], more]), pts[3551], forms,
             tol, **kw)


# points that gather in a few leaves take a warp per box, and more boxes than
# warps are walked over
@pytest.mark.parametrize("kw", [{}, dict(skip_empty=True), dict(sparse=True)])
def test_p2m_clustered_points_take_a_warp_per_box(gpu_lib, kw):
    rng = np.random.default_rng(6)
    n, order = 40000, 8
    pts = np.clip(0.25 + 0.03 * rng.standard_normal((n, 3)), -0.5, 0.5)
    pts[:n // 4] = rng.uniform(-0.5, 0.5, (n // 4, 3))
    q = rng.standard_normal(n)
    got = {}
    for depth in (4, 5):
        cfg = engine.SolverConfig(LAP, depth, [0] + [order] * depth, [0] + [order] * depth, 0.0,
                                  (-0.51,) * 3, 1.02, engine.FP64, **kw)
        with engine.Solver(cfg) as s:
            s.set_sources(pts).set_strengths(q).set_targets(pts).leaf_expansions()
            assert s.p2m_form() == 32
            if depth == 5:
                s.upward_pass(5)
            got[depth] = s.coefficients(4)[0]
    # the shift of exact expansions is exact in the degrees kept
    assert np.linalg.norm(got[5] - got[4]) < 1e-12 * np.linalg.norm(got[4])


# (the sums of a few hundred terms: ten units)
@pytest.mark.parametrize("precision,tol", [(engine.FP64, 2e-14), (engine.FP32, 4e-6)])
@pytest.mark.parametrize("problem", [LAP, HELM])
@pytest.mark.parametrize("order,dipoles", [(2, False), (6, True), (14, False), (14, True), (24, False)])
@pytest.mark.parametrize("depth", [2, 3])
def test_p2m_shared(gpu_lib, problem, precision, tol, order, dipoles, depth):
    pts = np.random.default_rng(order).uniform(-0.5, 0.5, (48 * 8 ** depth, 3))
    _compare(problem, precision, order, dipoles, depth, pts, np.full(3, -0.3), (32, 128), tol)


# leaves of more than 32 points need eight times the groups, and none may hold
# more than 128 (one leaf of each of as many parents); against the depth above
@pytest.mark.parametrize("full,groups,form", [(33, 28415, 32), (33, 28416, 8), (128, 28416, 8),
                                              (129, 28416, 32)])
def test_p2m_many_groups(gpu_lib, full, groups, form):
    rng = np.random.default_rng(7)
    ijk = np.stack(np.meshgrid(*[np.arange(32)] * 3, indexing="ij"), -1).reshape(-1, 3)
    ijk = rng.permutation(ijk)[:groups]                  # parents of depth 6's leaves
    width = W5 / 2
    pts = (2 * ijk + 0.4) * width - 0.51
    pts = np.concatenate([pts, (2 * ijk[0] + rng.uniform(0.1, 0.9, (full - 1, 3))) * width - 0.51])
    q = rng.standard_normal(len(pts))

    def level5(depth, **kw):
        orders = [0] + [6] * depth
        cfg = engine.SolverConfig(LAP, depth, orders, list(orders), 0.0, (-0.51,) * 3, 1.02,
                                  engine.FP64, **kw)
        with engine.Solver(cfg) as s:
            s.set_sources(pts).set_strengths(q).set_targets(pts).leaf_expansions()
            assert depth == 5 or s.p2m_form() == form
            if depth == 6:
                s.upward_pass(6)
            return s.coefficients(5)[0]

    want = level5(5)
    for kw in ({}, dict(sparse=True)):
        got = level5(6, **kw)
        assert np.linalg.norm(got - want) < 1e-12 * np.linalg.norm(want)
