"""Few leaves of many points: the P2M by a block per leaf and the near field by several blocks per leaf, at leaf sizes
around the groups of 32 points and the tiles of 256 sources, with fewer tiles than blocks, several targets' rounds of a
block, empty leaves and lists longer than a batch's tiles."""
import numpy as np
import pytest

from bachelors_b200 import Plan, geometry as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n,m,cap", [(512, 1, 600), (513, 65, 600), (2305, 700, 3000), (4103, 301, 700), (9001, 2003, 500),
                                     (20000, 97, 257)])
# the rounding of the whole pipeline against the oracle on the same inputs, as in the parity tests
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
def test_large_leaves_match_oracle(n, m, cap, precision, tol):
    rng = np.random.default_rng(n)
    xyz = np.concatenate([rng.uniform(-1, 1, (n - n // 4, 3)), rng.normal(size=(n // 4, 3)) * 0.05 + 0.6])
    w, J, tgt = rng.uniform(0.5, 1, n), rng.normal(size=(n, 3)), rng.uniform(-1.2, 1.2, (m, 3))
    if precision == "fp32":
        xyz, w, J, tgt = (v.astype(np.float32).astype(np.float64) for v in (xyz, w, J, tgt))
    c, H = G.root_cube(xyz, tgt)
    Bo, Ao, so = O.fmm(7, cap, xyz, w, J, tgt, c, H, want_A=True)
    plan = Plan(order=7, leaf_capacity=cap, precision=precision)
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    for want in (1, 2, 3):
        B, A = plan.solve(1.0, want)
        assert B is None or rel(B, Bo) < tol
        assert A is None or rel(A, Ao) < tol
    assert plan.stats()["nodes"] == so["nodes"]
    plan.close()


@pytest.mark.parametrize("n,m,cap,short", [(20000, 3000, 8, True), (120000, 12000, 96, False)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
def test_near_block_sizes(n, m, cap, short, precision, tol):
    """More boxes than run at once, short and long lists: both sizes of the near field's blocks, leaves whose targets do
    and do not divide the block."""
    rng = np.random.default_rng(n)
    xyz, w, J = rng.uniform(-1, 1, (n, 3)), rng.uniform(0.5, 1, n), rng.normal(size=(n, 3))
    tgt = np.concatenate([rng.uniform(-1, 1, (m - 1000, 3)), rng.uniform(0.1, 0.3, (1000, 3))])
    if precision == "fp32":
        xyz, w, J, tgt = (v.astype(np.float32).astype(np.float64) for v in (xyz, w, J, tgt))
    c, H = G.root_cube(xyz, tgt)
    Bo, Ao, so = O.fmm(4, cap, xyz, w, J, tgt, c, H, want_A=True)
    plan = Plan(order=4, leaf_capacity=cap, precision=precision)
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    B, _ = plan.solve(1.0, 1)
    assert rel(B, Bo) < tol
    B, A = plan.solve(1.0, 3)
    st = plan.stats()
    plan.close()
    assert rel(B, Bo) < tol and rel(A, Ao) < tol
    assert st["nodes"] == so["nodes"] > 16 * 148
    assert (st["p2p_pairs"] / st["nodes"] * n / st["nodes"] < 256) == short
