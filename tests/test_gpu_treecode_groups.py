"""The treecode's groups of query points: many points (sorted, up to 32 a block) against the same points asked a few
at a time (a block each), and against the direct sum where a point sits on a source or far outside the tree."""
import numpy as np
import pytest

from bachelors_b200 import MultipoleSolver, Plan, geometry as G

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


# (orders 1 and 16 are the smallest and largest tables; 20,011 points over few boxes make groups of 32, 3,001 over
# more boxes smaller ones)
@pytest.mark.parametrize("p,cap,m", [(1, 400, 20011), (10, 400, 20011), (16, 400, 2999), (7, 40, 3001)])
@pytest.mark.parametrize("flags", [{}, {"reference_near": True, "fd_curl": True}])
def test_groups_equal_single_points(p, cap, m, flags):
    xyz, w, J = G.torus(40, 16, 8, 2.0, 0.5)
    s = MultipoleSolver((xyz, w, J), quadratureOctreeLeafCapacity=cap, order=p, precision="fp64")
    s.calcMultipoleExpansionsAtLeaves()
    pts = G.uniform_points(m, -3, 3, p)
    pts[:5] = [[0, 0, 0], [50, 1, 2], [-9, 0, 0], [2.0, 0, 0.1], [0, -2.2, 0]]
    B, A = s.plan.treecode(pts, 1.0, 3, **flags)
    pick = np.concatenate([np.arange(5), np.random.default_rng(1).choice(m, 90, replace=False)])
    few = [s.plan.treecode(pts[pick[i:i + 7]], 1.0, 3, **flags) for i in range(0, len(pick), 7)]
    # the same boxes and harmonics in another order of summation; the central differences divide by 2e-3
    tol = 1e-10 if flags else 1e-12
    assert rel(B[pick], np.concatenate([f[0] for f in few])) < tol
    assert rel(A[pick], np.concatenate([f[1] for f in few])) < 1e-12
    s.plan.close()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-6), ("fp32", 1e-5)])
def test_points_on_sources_and_far_away(precision, tol):
    """Own source skipped; far points meet the root box alone. The expansion error at p = 12 is below 1e-6."""
    xyz, w, J = G.torus(32, 12, 6, 2.0, 0.5)
    pts = np.concatenate([xyz[::37], [[30.0, 2, 1], [0, 0, 90]]])
    if precision == "fp32":
        xyz, w, J, pts = (v.astype(np.float32).astype(np.float64) for v in (xyz, w, J, pts))
    s = MultipoleSolver((xyz, w, J), quadratureOctreeLeafCapacity=60, order=12, precision=precision)
    s.calcMultipoleExpansionsAtLeaves()
    got = s.calcB(1.0, pts)
    ref = Plan(order=1, leaf_capacity=1 << 30, precision="fp64")
    ref.set_sources(xyz, w, J)
    ref.set_targets(pts)
    want = ref.direct(1.0, 1)[0]
    assert rel(got, want) < tol
    ref.close()
    s.plan.close()


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_calls_on_two_streams(precision):
    """Queries of different sizes, one after the other on two streams without a wait by the caller: the plan's scratch
    (the points' order, the curl table) is never one call's while another's kernel reads it. The results equal those
    of the same calls on one stream, bit for bit."""
    import torch
    dt = torch.float32 if precision == "fp32" else torch.float64
    xyz, w, J = (torch.tensor(v, dtype=dt, device="cuda") for v in G.torus(64, 24, 12, 2.0, 0.5))
    pts = [torch.tensor(G.uniform_points(m, -3, 3, m), dtype=dt, device="cuda") for m in (4099, 30011, 9001, 50021, 7)]

    def queries(streams):
        s = MultipoleSolver((xyz, w, J), quadratureOctreeLeafCapacity=500, order=8, precision=precision)
        s.calcMultipoleExpansionsAtLeaves()
        torch.cuda.synchronize()
        out = []
        for i, p in enumerate(pts):
            with torch.cuda.stream(streams[i % len(streams)]):
                out.append(s.calcB(1.0, p))
        torch.cuda.synchronize()
        out = [v.cpu().numpy() for v in out]
        s.plan.close()
        return out

    for a, b in zip(queries([torch.cuda.current_stream()]), queries([torch.cuda.Stream(), torch.cuda.Stream()])):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("then", ["new sources", "new strengths", "graph", "direct", "autotune"])
def test_next_call_on_another_stream(precision, then):
    """A query still running on one stream when the plan's next call comes on another and changes the sources, the
    tree or the multipoles: the query's result stays what it is alone, bit for bit."""
    import torch
    dt = torch.float32 if precision == "fp32" else torch.float64
    cuda = lambda a: torch.tensor(a, dtype=dt, device="cuda")
    xyz, w, J = (cuda(v) for v in G.torus(64, 24, 12, 2.0, 0.5))
    rng = np.random.default_rng(4)
    other = [cuda(rng.uniform(-1, 1, (3001, 3))), cuda(rng.uniform(1, 2, 3001)), cuda(rng.normal(size=(3001, 3)))]
    pts, tgt = cuda(G.uniform_points(50021, -3, 3, 1)), cuda(G.uniform_points(300, -3, 3, 2))
    plan = Plan(order=8, leaf_capacity=300, precision=precision)
    plan.set_sources(xyz, w, J)
    plan.set_targets(tgt)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(2):
        plan.set_sources(xyz, w, J)
        plan.set_targets(tgt)
        plan.solve(1.0, 1)
        if then == "graph":
            plan.graph_capture(1)
        alone = plan.treecode(pts, 1.0, 1)[0].clone()
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            got = plan.treecode(pts, 1.0, 1)[0]
        with torch.cuda.stream(b):
            if then == "new sources":
                plan.set_sources(*other)
                plan.build_tree()
                plan.upward()
            elif then == "new strengths":
                plan.update_sources(w * 3, J)
                plan.upward()
            elif then == "graph":
                plan.graph_launch(1.0)
            elif then == "direct":
                plan.set_targets(tgt + 1)
                plan.direct(1.0, 1)
            else:
                plan.autotune()
        torch.cuda.synchronize()
        assert torch.equal(got, alone)
    plan.close()


@pytest.mark.parametrize("p,cap,m", [(1, 10, 40009), (5, 20, 20011), (9, 30, 1301)])
def test_groups_over_many_boxes(p, cap, m):
    """Groups larger than the points a box has: most boxes want few of a block's points."""
    test_groups_equal_single_points(p, cap, m, {})
