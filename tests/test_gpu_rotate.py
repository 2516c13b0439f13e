"""Translations through the z axis (M2L, M2M, L2L on the CUDA cores) against the oracle's dense ones: every
kind of order (block sizes that fill the four-output groups and that do not, odd and even), few and many boxes
(chunks of pairs that are full, that have a remainder and that hold one pair), both precisions."""
import numpy as np
import pytest

from bachelors_b200 import Plan, geometry as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


def solve(p, cap, precision, xyz, w, J, tgt, want=3, **kw):
    plan = Plan(order=p, leaf_capacity=cap, precision=precision, **kw)
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    out = [np.asarray(v, np.float64) for v in plan.solve(1.0, want) if v is not None]
    st = plan.stats()
    plan.close()
    return out, st


@pytest.mark.parametrize("p,cap", [(1, 6), (2, 6), (3, 8), (4, 8), (5, 8), (6, 8), (7, 10), (8, 10), (9, 10), (11, 12),
                                   (12, 16), (13, 16), (15, 16), (16, 16)])
def test_translations_match_oracle(p, cap):
    xyz, w, J = G.torus(24, 8, 5, 2.0, 0.5)
    tgt = G.uniform_points(701, -3, 3, p)
    c, H = G.root_cube(xyz, tgt)
    Bo, Ao, so = O.fmm(p, cap, xyz, w, J, tgt, c, H, want_A=True)
    (B, A), st = solve(p, cap, "fp64", xyz, w, J, tgt)
    assert st["nodes"] == so["nodes"] and st["v_pairs"] > 0
    assert rel(B, Bo) < 1e-12 and rel(A, Ao) < 1e-12
    # FP32: the same FP32 inputs in the oracle, rounding of ~1e2 accumulated terms of 2^-24 each
    x32, w32, J32, t32 = (v.astype(np.float32) for v in (xyz, w, J, tgt))
    c, H = G.root_cube(x32.astype(np.float64), t32.astype(np.float64))
    Bo, Ao, _ = O.fmm(p, cap, *(v.astype(np.float64) for v in (x32, w32, J32, t32)), c, H, want_A=True)
    (B, A), _ = solve(p, cap, "fp32", x32, w32, J32, t32)
    assert rel(B, Bo) < 1e-5 and rel(A, Ao) < 1e-5


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
def test_one_pair_and_uneven_levels(precision, tol):
    """Two far clusters (one box pair a level) and a dense cluster that deepens one branch of the tree."""
    rng = np.random.default_rng(3)
    far = np.concatenate([rng.uniform(-0.02, 0.02, (7, 3)) + 2.9, rng.uniform(-0.02, 0.02, (7, 3)) - 2.9])
    dense = rng.normal(size=(400, 3)) * 0.01 + 1.0
    xyz = np.concatenate([far, dense])
    w = rng.uniform(0.5, 1.5, len(xyz))
    J = rng.normal(size=xyz.shape)
    tgt = np.concatenate([far[:5] + 0.05, dense[:37] + 0.02, rng.uniform(-3, 3, (21, 3))])
    if precision == "fp32":
        xyz, w, J, tgt = (v.astype(np.float32).astype(np.float64) for v in (xyz, w, J, tgt))
    c, H = G.root_cube(xyz, tgt)
    Bo, Ao, so = O.fmm(9, 8, xyz, w, J, tgt, c, H, want_A=True)
    (B, A), st = solve(9, 8, precision, xyz, w, J, tgt)
    assert st["nodes"] == so["nodes"]
    assert rel(B, Bo) < tol and rel(A, Ao) < tol


@pytest.mark.parametrize("p,precision", [(1, "fp32"), (1, "fp64"), (4, "fp32"), (10, "fp64")])
@pytest.mark.parametrize("cutoff", ["p", "p + 1", "2 p", "none"])
def test_degree_cutoff_is_the_tensor_cores(p, precision, cutoff):
    """m2l_tc_degree_cutoff belongs to the tensor-core M2L: a CUDA-core plan applies its full operator whatever the
    value, bit for bit."""
    xyz, w, J = G.torus(24, 8, 5, 2.0, 0.5)
    tgt = G.uniform_points(301, -3, 3, p)
    if precision == "fp32":
        xyz, w, J, tgt = (v.astype(np.float32) for v in (xyz, w, J, tgt))
    (full,), st = solve(p, 8, precision, xyz, w, J, tgt, want=1)
    (cut,), _ = solve(p, 8, precision, xyz, w, J, tgt, want=1,
                      m2l_degree_cutoff={"p": p, "p + 1": p + 1, "2 p": 2 * p, "none": -1}[cutoff])
    assert st["v_pairs"] > 0
    np.testing.assert_array_equal(cut, full)
