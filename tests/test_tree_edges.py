"""Tree build at the edges of its sorts (one CTA up to 4096 points, tiles of
2048 above) and of its level-at-once refinement: permutation and boxes of every
level bit-exact with the CPU restatement."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle_api import level_box_offsets
from wbfmm_b200 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 1024, 1025, 4095, 4096, 4097, 6144, 6145, 530000])
@pytest.mark.parametrize("kind", ["cube", "few"])
def test_tree(restatement, gpu_lib, n, kind):
    rng = np.random.default_rng(n)
    if kind == "cube":
        pts = rng.uniform(-0.5, 0.5, (n, 3))
    else:   # many equal keys, most boxes empty, points in the last octants
        pts = rng.choice(rng.uniform(0.2, 0.499, (7, 3)), n)
    depth = 4
    x0, D = np.array([-0.51, -0.51, -0.51]), 1.02
    want, boxes = restatement.tree_build(x0, D, depth, pts)
    cfg = engine.SolverConfig(engine.LAPLACE, depth, [0] + [2] * depth, [0] + [2] * depth, 0.0,
                              tuple(x0), D)
    with engine.Solver(cfg) as s:
        s.set_sources(pts)
        off = level_box_offsets(depth)
        for lv in range(depth + 1):
            ip, bi, bn = s.tree(lv)
            assert np.array_equal(ip, want)
            sl = slice(off[lv], off[lv] + 8 ** lv)
            assert np.array_equal(bi, boxes[sl, 0]) and np.array_equal(bn, boxes[sl, 1])


# a refused set_sources (a point on the cube's face) leaves the sources in
# place: new strengths give the fields they gave before
@pytest.mark.parametrize("n", [3000, 6000])            # both sorts
@pytest.mark.parametrize("refused", ["same", "fewer", "more"])
def test_refused_sources_keep_the_tree(gpu_lib, n, refused):
    rng = np.random.default_rng(n)
    pts, q = rng.uniform(-0.5, 0.5, (n, 3)), rng.standard_normal(n)
    bad = rng.uniform(-0.5, 0.5, ({"same": n, "fewer": n // 2, "more": 2 * n}[refused], 3))
    bad[7, 1] = -0.51
    cfg = engine.SolverConfig(engine.LAPLACE, 3, [0, 6, 6, 6], [0, 6, 6, 6], 0.0, (-0.51,) * 3, 1.02,
                              engine.FP64, engine.POTENTIAL | engine.GRADIENT)
    with engine.Solver(cfg) as s:
        want = s.set_sources(pts).set_strengths(q).set_targets(pts).run().field()
        with pytest.raises(engine.WbfmmError):
            s.set_sources(bad)
        got = s.set_strengths(q).run().field()
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
        ip, _, bn = s.tree(3)
        assert np.array_equal(np.sort(ip), np.arange(n)) and bn.sum() == n
