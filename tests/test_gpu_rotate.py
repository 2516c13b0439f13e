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


def memory_used(plan_args, xyz, w, J, tgt):
    """Device memory a plan with a solve behind it holds, beyond its first solve of a little problem."""
    import torch
    plan = Plan(**plan_args)
    plan.set_sources(xyz[:64], w[:64], J[:64])
    plan.set_targets(tgt[:64])
    plan.solve(1.0, 1)
    free = torch.cuda.mem_get_info()[0]
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    plan.solve(1.0, 1)
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    plan.close()
    return used


@pytest.mark.parametrize("p,n,leaf,precision", [(3, 250007, 2, "fp32"), (3, 150001, 2, "fp64"), (13, 60013, 3, "fp32"),
                                                (13, 40009, 3, "fp64"), (9, 30011, 4, "fp32"), (16, 9001, 20, "fp64")])
def test_whole_and_shared_tiles(monkeypatch, p, n, leaf, precision):
    """Trees from a few tiles to several rounds of blocks (whole tiles, shared ones, parents and children in more tiles
    than blocks): the same sums with every tile a block's own, and the direct sum at some targets."""
    rng = np.random.default_rng(n)
    dt = np.float32 if precision == "fp32" else np.float64
    # uneven density, so that the tiles' operators differ
    xyz = np.concatenate([rng.uniform(-1, 1, (n - n // 3, 3)), rng.normal(size=(n // 3, 3)) * 0.1 + 0.5]).astype(dt)
    w, J = rng.uniform(0.5, 1.5, n).astype(dt), rng.normal(size=(n, 3)).astype(dt)
    tgt = np.concatenate([xyz[::2] + dt(0.001), rng.uniform(-1, 1, (n // 2, 3)).astype(dt)]).astype(dt)
    (B, A), st = solve(p, leaf, precision, xyz, w, J, tgt)
    monkeypatch.setenv("FMM_SPLIT_SUMS", "0")
    (Bo, Ao), _ = solve(p, leaf, precision, xyz, w, J, tgt)
    # the same terms in another order: ~1e3 of them, 2^-24 (2^-53) each
    tol = 1e-5 if precision == "fp32" else 1e-13
    assert rel(B, Bo) < tol and rel(A, Ao) < tol
    pick = rng.choice(len(tgt), 50, replace=False)
    plan = Plan(order=2, precision=precision)
    plan.set_sources(xyz, w, J)
    D = plan.direct_fp64(tgt[pick])
    plan.close()
    assert rel(B[pick], D) < {3: 5e-2, 9: 2e-3, 13: 2e-4, 16: 1e-4}[p]


@pytest.mark.parametrize("p,precision", [(9, "fp32"), (12, "fp32"), (9, "fp64"), (16, "fp64")])
def test_scratch_is_bounded(monkeypatch, p, precision):
    """The room for split sums: at most 75 MB beside what the plan needs without them (16 MB for the granularity of
    allocations)."""
    rng = np.random.default_rng(p)
    n = 60000
    xyz, w, J = rng.uniform(-1, 1, (n, 3)), rng.uniform(0.5, 1.5, n), rng.normal(size=(n, 3))
    args = dict(order=p, leaf_capacity=20, precision=precision)
    with_room = memory_used(args, xyz, w, J, xyz)
    monkeypatch.setenv("FMM_SPLIT_SUMS", "0")
    without = memory_used(args, xyz, w, J, xyz)
    assert with_room - without < (75 + 16) << 20
