"""Direct lists a warp per leaf: the direct pairs of trees with very unequal leaves (one list of thousands of small boxes
below a large neighbour, long chains of levels) counted against the oracle's tree, and the field against it."""
import numpy as np
import pytest

from bachelors_b200 import Plan
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("kind,cap", [("dense corner", 2), ("chain", 1), ("uniform", 3), ("one box", 5000)])
def test_direct_pairs_of_uneven_trees(kind, cap):
    rng = np.random.default_rng(4)
    if kind == "dense corner":
        # 3,000 sources against the face of a large, almost empty box: its leaf meets every small box beyond the face
        xyz = np.concatenate([rng.uniform([0.001, -0.5, -0.5], [0.02, 0.5, 0.5], (3000, 3)), [[-0.9, -0.9, -0.9]]])
        tgt = np.concatenate([rng.uniform([-0.5, -0.5, -0.5], [-0.001, 0.5, 0.5], (2, 3)), [[1.0, 1.0, 1.0]]])
    elif kind == "chain":
        # points halving their distance to a corner: a level per pair of points
        xyz = np.array([[2.0 ** -i] * 3 for i in range(18)]) * [1.0, 0.99, 0.98]
        tgt = xyz * 0.97
    else:
        xyz = rng.uniform(-1, 1, (700, 3))
        tgt = rng.uniform(-1, 1, (300, 3))
    w, J = rng.uniform(0.5, 1, len(xyz)), rng.normal(size=xyz.shape)
    lo, hi = np.min(np.r_[xyz, tgt], axis=0), np.max(np.r_[xyz, tgt], axis=0)
    c, H = 0.5 * (lo + hi), 0.5 * float(np.max(hi - lo)) * (1 + 2.0 ** -20) + 1e-300
    Bo, _, so = O.fmm(8, cap, xyz, w, J, tgt, c, H)
    plan = Plan(order=8, leaf_capacity=cap, precision="fp64")
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    B, _ = plan.solve(1.0, 1)
    st = plan.stats()
    assert (st["nodes"], st["p2p_interactions"]) == (so["nodes"], so["direct_pairs"])
    assert rel(B, Bo) < 1e-12
    plan.close()
