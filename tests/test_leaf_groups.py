"""P2M with a few points per leaf (8 lanes per box) against a warp per box: the
rule changes sides at 12 points per leaf on average (from 24 leaves per SM), so
a problem on it and the same problem with one more source of strength zero take
the two forms."""
from __future__ import annotations

import numpy as np
import pytest

from wbfmm_b200 import engine

pytestmark = pytest.mark.gpu


# both forms add a leaf's at most few dozen terms of like size in another
# order: a few units of rounding of the level's norm
@pytest.mark.parametrize("precision,tol", [(engine.FP64, 1e-14), (engine.FP32, 2e-6)])
@pytest.mark.parametrize("problem", [engine.LAPLACE, engine.HELMHOLTZ])
@pytest.mark.parametrize("order", [2, 6, 14, 17])
@pytest.mark.parametrize("dipoles", [False, True])
def test_p2m_forms(gpu_lib, problem, precision, tol, order, dipoles):
    rng = np.random.default_rng(order)
    depth, n = 4, 12 * 4096
    w = 2 if problem == engine.HELMHOLTZ else 1
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

    few, whole = leaves(0), leaves(1)
    assert np.linalg.norm(few - whole) < tol * np.linalg.norm(whole)
