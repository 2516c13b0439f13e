"""Sources and targets sorted together: sizes on both sides of the rule (more than 2,500 points each, 2^19 in all), with
equal points among the two sets. (Several coils, whose bits lie below the mark: test_gpu_batch.py.)"""
import numpy as np
import pytest

from bachelors_b200 import Plan, geometry as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n,m", [(2500, 2501), (2501, 2500), (2501, 2501), (3000, 40000)])
def test_tree_matches_oracle(n, m):
    rng = np.random.default_rng(n + m)
    xyz, w, J = rng.uniform(-1, 1, (n, 3)), rng.uniform(0.5, 1, n), rng.normal(size=(n, 3))
    tgt = np.concatenate([xyz[::7], rng.uniform(-1.1, 1.1, (m - len(xyz[::7]), 3))])
    c, H = G.root_cube(xyz, tgt)
    Bo, _, so = O.fmm(4, 20, xyz, w, J, tgt, c, H)
    plan = Plan(order=4, leaf_capacity=20, precision="fp64")
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    B, _ = plan.solve(1.0, 1)
    st = plan.stats()
    plan.close()
    assert (st["nodes"], st["p2p_interactions"]) == (so["nodes"], so["direct_pairs"])
    assert rel(B, Bo) < 1e-12          # the same tree and FP64 arithmetic


@pytest.mark.parametrize("n,m", [((1 << 18) - 1, (1 << 18) + 1), (1 << 18, (1 << 18) + 1)])
def test_largest_joint_size(n, m):
    """At the limit and one point past it."""
    rng = np.random.default_rng(5)
    xyz, w, J = rng.uniform(-1, 1, (n, 3)), rng.uniform(0.5, 1, n), rng.normal(size=(n, 3))
    tgt = rng.uniform(-1, 1, (m, 3))
    plan = Plan(order=8, leaf_capacity=64, precision="fp64")
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    B, _ = plan.solve(1.0, 1)
    Bd = plan.direct_fp64(tgt[:64])
    plan.close()
    assert rel(B[:64], Bd) < 1e-4       # the truncation at order 8

