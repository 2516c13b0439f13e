"""The direct sum with its sources split over blocks and without a tree: sizes around the block (128 targets) and the
smallest part (512 sources), both precisions, B and A, coils, and what a plan accepts after fmm_direct."""
import numpy as np
import pytest

from bachelors_b200 import FmmError, Plan, geometry as G

pytestmark = pytest.mark.gpu


def reference(xyz, w, J, tgt, dtype=np.float64):
    """B and A in FP64 from strengths w J rounded to the plan's type, as the plan packs them."""
    d = tgt[:, None, :] - xyz[None, :, :]
    r2 = (d ** 2).sum(-1)
    ri = np.where(r2 > 0, 1 / np.sqrt(np.where(r2 > 0, r2, 1)), 0)
    q = (w.astype(dtype)[:, None] * J.astype(dtype)).astype(np.float64)
    B = np.cross(q[None], d)
    c = 4 * 3.14159265359
    return 1.2566370614e-6 / c * (B * (ri ** 3)[..., None]).sum(1), (q[None] * ri[..., None]).sum(1) / c


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n,m", [(1, 1), (511, 127), (512, 128), (1023, 129), (1024, 5), (5003, 300)])
# FP32: n terms of 2^-24 each in blocks of at most a few thousand, against the same FP32 inputs
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 3e-5)])
def test_direct_sizes(n, m, precision, tol):
    rng = np.random.default_rng(n + m)
    xyz, w, J = rng.uniform(-1, 1, (n, 3)), rng.uniform(0.5, 1, n), rng.normal(size=(n, 3))
    tgt = rng.uniform(-1.5, 1.5, (m, 3))
    if m > 1:
        tgt[0] = xyz[0]                                  # a coincident pair
    if precision == "fp32":
        xyz, w, J, tgt = (v.astype(np.float32).astype(np.float64) for v in (xyz, w, J, tgt))
    plan = Plan(order=2, leaf_capacity=64, precision=precision)
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    Bo, Ao = reference(xyz, w, J, tgt, np.float32 if precision == "fp32" else np.float64)
    for want in (1, 2, 3):
        B, A = plan.direct(1.0, want)
        assert B is None or rel(B, Bo) < tol
        assert A is None or rel(A, Ao) < tol
    assert rel(plan.direct_fp64(tgt), Bo) < 1e-12
    plan.solve(1.0, 1)                                  # the same sums over the tree's order of the sources
    assert rel(plan.direct(1.0, 1)[0], Bo) < tol
    plan.close()


def test_after_direct():
    xyz, w, J = G.torus(16, 8, 4)
    tgt = G.uniform_points(100, -3, 3, 1)
    plan = Plan(order=4, leaf_capacity=16, precision="fp64")
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    with pytest.raises(FmmError):
        plan.upward()                                   # no tree
    plan.direct(1.0, 1)
    nodes = plan.stats()["nodes"]
    plan.upward()                                       # fmm_direct stands for the tree build
    plan.downward()
    B, _ = plan.evaluate(1.0, 1)
    S, _ = plan.solve(1.0, 1)
    assert np.array_equal(B, S) and plan.stats()["nodes"] == nodes
    plan.set_targets(tgt[:50])
    with pytest.raises(FmmError):
        plan.upward()                                   # new inputs: not any more
    plan.close()
    # coils see only their own sources
    plan = Plan(order=2, precision="fp64")
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    plan.set_coils([0, 200, 200, len(w)], [0, 30, 60, 100])
    B, _ = plan.direct(1.0, 1)
    assert rel(B[:30], reference(xyz[:200], w[:200], J[:200], tgt[:30])[0]) < 1e-12
    assert not B[30:60].any()
    assert rel(B[60:], reference(xyz[200:], w[200:], J[200:], tgt[60:])[0]) < 1e-12
    plan.close()


def _cuda(*arrays, dtype):
    import torch
    return [torch.tensor(a, dtype=dtype, device="cuda") for a in arrays]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("then", ["solve", "new sources", "new targets", "subset"])
def test_next_call_on_another_stream(precision, then):
    """A direct sum without a tree, still running on one stream when the plan's next call comes on another: that call
    changes the sources' order (a tree build, another direct sum), the inputs, or runs a sum of its own, and the first
    one's result stays what it is alone, bit for bit."""
    import torch
    dt = torch.float64 if precision == "fp64" else torch.float32
    rng = np.random.default_rng(8)
    n, m = 150001, 9001
    xyz, w, J, tgt = _cuda(rng.uniform(-1, 1, (n, 3)), rng.uniform(0.5, 1, n), rng.normal(size=(n, 3)),
                           rng.uniform(-2, 2, (m, 3)), dtype=dt)
    other = _cuda(rng.uniform(3, 4, (n, 3)), rng.uniform(0.5, 1, n), rng.normal(size=(n, 3)), dtype=dt)
    plan = Plan(order=3, leaf_capacity=200, precision=precision)
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    alone = plan.direct(1.0, 1)[0].clone()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(3):
        plan.set_sources(xyz, w, J)
        plan.set_targets(tgt)
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            got = plan.direct(1.0, 1)[0]
        with torch.cuda.stream(b):
            if then == "solve":
                plan.solve(1.0, 1)
            elif then == "new sources":
                plan.set_sources(*other)
                plan.build_tree()
            elif then == "new targets":
                plan.set_targets(tgt.clone())
                plan.build_tree()
            else:
                plan.direct_fp64(rng.uniform(-2, 2, (3, 3)))
        torch.cuda.synchronize()
        assert torch.equal(got, alone)
    plan.close()


def test_captured_by_the_caller():
    """A direct sum over a plan's tree, captured into a graph of the caller's and replayed; the plan goes on."""
    import torch
    rng = np.random.default_rng(9)
    xyz, w, J, tgt = _cuda(rng.uniform(-1, 1, (5000, 3)), rng.uniform(0.5, 1, 5000), rng.normal(size=(5000, 3)),
                           rng.uniform(-2, 2, (300, 3)), dtype=torch.float64)
    plan = Plan(order=3, leaf_capacity=100, precision="fp64")
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    plan.solve(1.0, 1)
    want = plan.direct(1.0, 1)[0].clone()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        got = plan.direct(1.0, 1)[0]
    for _ in range(2):
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    plan.build_tree()
    assert torch.equal(plan.direct(1.0, 1)[0], want)
    plan.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_own_source_is_skipped_whatever_its_strength(precision, bad):
    """A target on a source whose strength is no number, in a coil of its own: the pair is skipped, so the other
    sources alone make its field; targets off that source see the value. The treecode's leaves do the same."""
    rng = np.random.default_rng(10)
    dt = np.float32 if precision == "fp32" else np.float64
    xyz, w, J = rng.uniform(-1, 1, (700, 3)).astype(dt), rng.uniform(0.5, 1, 700).astype(dt), rng.normal(size=(700, 3)).astype(dt)
    J[37] = bad
    tgt = np.concatenate([xyz[37:38], xyz[37:38], [[2.0, 0, 0]]]).astype(dt)
    rest = np.arange(700) != 37
    Bo, Ao = reference(*(v.astype(np.float64) for v in (xyz[rest], w[rest], J[rest], tgt)), dt)
    plan = Plan(order=2, leaf_capacity=1000, precision=precision)
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    tol = 1e-12 if precision == "fp64" else 3e-5
    for want in (1, 2, 3):
        B, A = plan.direct(1.0, want)
        assert B is None or (rel(B[:2], Bo[:2]) < tol and not np.isfinite(B[2]).all())
        assert A is None or (rel(A[:2], Ao[:2]) < tol and not np.isfinite(A[2]).all())
    assert rel(plan.direct_fp64(tgt[:2]), Bo[:2]) < 1e-12
    plan.build_tree()
    plan.upward()
    B, A = plan.treecode(tgt[:2], 1.0, 3)
    assert rel(B, Bo[:2]) < tol and rel(A, Ao[:2]) < tol
    plan.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_sources_packed_once_follow_the_inputs(precision):
    """The sources are packed by the first of several direct sums and again when anything they depend on changes: every
    sum equals that of a new plan with the same inputs, bit for bit."""
    dt = np.float32 if precision == "fp32" else np.float64
    rng = np.random.default_rng(11)
    n, m = 1500, 40
    sets = [[v.astype(dt) for v in (rng.uniform(-1, 1, (n, 3)), rng.uniform(0.5, 1, n), rng.normal(size=(n, 3)))] for _ in range(2)]
    tgts = [rng.uniform(-2, 2, (m, 3)).astype(dt) for _ in range(2)]

    def fresh(s, t, coils=None):
        plan = Plan(order=3, leaf_capacity=50, precision=precision)
        plan.set_sources(*s)
        plan.set_targets(t)
        if coils:
            plan.set_coils(*coils)
        out = plan.direct(1.0, 1)[0].copy()
        plan.close()
        return out

    plan = Plan(order=3, leaf_capacity=50, precision=precision)
    plan.set_sources(*sets[0])
    plan.set_targets(tgts[0])
    for _ in range(3):
        assert np.array_equal(plan.direct(1.0, 1)[0], fresh(sets[0], tgts[0]))
    plan.set_targets(tgts[1])
    assert np.array_equal(plan.direct(1.0, 1)[0], fresh(sets[0], tgts[1]))
    plan.set_sources(*sets[1])
    assert np.array_equal(plan.direct(1.0, 1)[0], fresh(sets[1], tgts[1]))
    coils = ([0, 600, n], [0, 10, m])
    plan.set_coils(*coils)
    for _ in range(2):
        assert np.array_equal(plan.direct(1.0, 1)[0], fresh(sets[1], tgts[1], coils))
    plan.set_coils(None, None)
    assert np.array_equal(plan.direct(1.0, 1)[0], fresh(sets[1], tgts[1]))
    plan.solve(1.0, 1)                                   # the tree's order from here on
    tree = plan.direct(1.0, 1)[0].copy()
    assert rel(tree, fresh(sets[1], tgts[1]).astype(np.float64)) < (1e-12 if precision == "fp64" else 1e-5)
    assert np.array_equal(plan.direct(1.0, 1)[0], tree)
    plan.set_sources(*sets[0])                           # and back to the input order
    assert np.array_equal(plan.direct(1.0, 1)[0], fresh(sets[0], tgts[1]))
    plan.close()


def test_statistics_between_streams():
    """stats() after a direct sum builds the tree on the default stream; the phases then go on at once on another
    stream, and the sum still running on a third keeps its result."""
    import torch
    rng = np.random.default_rng(12)
    n, m = 60001, 3001
    xyz, w, J, tgt = _cuda(rng.uniform(-1, 1, (n, 3)), rng.uniform(0.5, 1, n), rng.normal(size=(n, 3)),
                           rng.uniform(-2, 2, (m, 3)), dtype=torch.float64)
    plan = Plan(order=4, leaf_capacity=60, precision="fp64")
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    want, alone = plan.solve(1.0, 1)[0].clone(), None
    for _ in range(2):
        plan.set_targets(tgt)
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.Stream()):
            D = plan.direct(1.0, 1)[0]
        st = plan.stats()
        with torch.cuda.stream(torch.cuda.Stream()):
            plan.upward()
            plan.downward()
            B = plan.evaluate(1.0, 1)[0]
        torch.cuda.synchronize()
        assert st["nodes"] > 1 and st["leaves"] > 1 and st["p2p_pairs"] > 0
        assert torch.equal(B, want)
        assert alone is None or torch.equal(D, alone)
        alone = D.clone()
    plan.close()
